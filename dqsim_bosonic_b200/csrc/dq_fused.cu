// dq_fused.cu — the tile-sweep engine: planner (host) and sweep kernel (sm_100a).
//
// The device side (tile geometry, the encoded program layout, the per-op
// register arithmetic and the per-CTA tile loop) is in dq_sweep.cuh.  The
// default launch runs 128 threads per CTA, three CTAs per SM.
//
// A sweep is a list of phases.  In a phase each thread holds 2^RB amplitudes
// in registers: the ones whose RB "register" local bits vary, at the thread
// bits given by its thread index.  Gate ops of the phase act on register
// bits only (dense 2x2 / 4x4, controlled X), so no data is exchanged between
// threads inside a phase; a new phase re-reads the tile with a new register
// assignment.  Per-gate arithmetic uses FMA (the tile path is held to the
// 1e-12 amplitude tolerance, the per-gate kernels to bit-exactness).
//
// Diagonal gates never need locality: they are accumulated on the host as a
// phase polynomial  c * prod_q w_q^{x_q} * prod_{q<r} w_qr^{x_q x_r}  and a
// FLUSH op applies all terms containing a qubit q right before the first
// non-diagonal gate on q.  A FLUSH multiplies the amplitudes with x_q = 1 by
// slot[s] * prod_{thread partners set} w * F[register index], where the
// per-tile factor slot[s] (q's linear term times its non-local partners
// whose bits are set in this tile's base index) is computed once per tile.
#include <cuda_runtime.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <mutex>
#include <string>
#include <vector>

#include "dq_common.cuh"
#include "dq_fused.cuh"
#include "dq_gates.hpp"
#include "dq_sweep.cuh"

namespace dq {

namespace {

// One persistent CTA per SM walks tiles blockIdx.x, + gridDim.x, ...
// S = 1 (128 threads): no prefetch, three CTAs per SM overlap each other's
// loads.  S = 2: the next tile's load is in flight while the current one is
// computed.  The sweep program is staged in shared memory once per launch
// (read from global memory per op instead, QFT30 ran 38% slower).
// FORM_H (every phase an H phase) and FORM_U (plain one-qubit ops only): built
// without the generic op interpreter (FORM_U: with its one-qubit part only),
// in few enough registers for four CTAs per SM.
template <int TB, int RB, int S, int RUNB, int FORM = FORM_ALL>
__global__ void __launch_bounds__(1 << TB, (S == 1 && TB == 7 ? (FORM != FORM_ALL ? 4 : 3)
                                                              : (TB + RB <= 11 ? 2 : 1)))
    k_sweep(double2* __restrict__ state, const uint8_t* __restrict__ gprog, uint32_t prog_bytes,
            uint32_t ntiles, long long synth) {
  constexpr int T = 1 << (TB + RB);
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* bufs = reinterpret_cast<double2*>(smraw);  // S tiles
  double2* slots = bufs + S * T;
  uint8_t* sprog = reinterpret_cast<uint8_t*>(slots + kMaxSlots);
  for (uint32_t i = threadIdx.x * 16u; i < prog_bytes; i += (1u << TB) * 16u)
    *reinterpret_cast<uint4*>(sprog + i) = __ldg(reinterpret_cast<const uint4*>(gprog + i));
  __syncthreads();
  sweep_tiles<TB, RB, S, RUNB, FORM>(state, sprog, ntiles, synth, bufs, slots, blockIdx.x, gridDim.x);
}

// Sweep k of many states in one launch: job j's tiles are split into chunks
// of chunk_tiles consecutive tiles and the CTAs take (job, chunk) work items
// in order; a CTA stages a job's program in shared memory when it moves to
// that job (a few KB per chunk of 2 MB of tiles).
template <int TB, int RB, int RUNB, int FORM = FORM_ALL>
__global__ void __launch_bounds__(1 << TB, TB == 7 ? (FORM != FORM_ALL ? 4 : 3) : 2)
    k_sweep_multi(const SweepJob* __restrict__ jobs, uint32_t njobs, uint32_t nchunks,
                  uint32_t chunk_tiles, uint32_t ntiles) {
  constexpr int T = 1 << (TB + RB);
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* bufs = reinterpret_cast<double2*>(smraw);
  double2* slots = bufs + T;
  uint8_t* sprog = reinterpret_cast<uint8_t*>(slots + kMaxSlots);
  const uint64_t work = (uint64_t)njobs * nchunks;
  uint64_t staged = ~0ULL;
  for (uint64_t w = blockIdx.x; w < work; w += gridDim.x) {
    const uint64_t j = w / nchunks;
    const SweepJob J = jobs[j];
    if (j != staged) {
      for (uint32_t i = threadIdx.x * 16u; i < J.prog_bytes; i += (1u << TB) * 16u)
        *reinterpret_cast<uint4*>(sprog + i) = __ldg(reinterpret_cast<const uint4*>(J.prog + i));
      __syncthreads();
      staged = j;
    }
    const uint32_t c = (uint32_t)(w % nchunks);
    const uint32_t t0 = c * chunk_tiles;
    const uint32_t t1 = min(t0 + chunk_tiles, ntiles);
    sweep_tiles<TB, RB, 1, RUNB, FORM>(J.state, sprog, t1, J.synth, bufs, slots, t0, 1);
    __syncthreads();
  }
}

// ---- relabel materialisation: paired-tile involution of bit positions ------------
//
// A bit-position involution tau (tau(tau(p)) = p) moves amplitude i to tau(i).
// With a local set L closed under tau, tile T maps onto tile tau(T), element
// e onto tau_L(e); one warp exchanges the pair (T, tau(T)) so the permutation
// is race-free in place.
//
// HBM bound: every amplitude is read and written once.  A tile is 2^8
// amplitudes (the four lowest positions, i.e. 256-byte runs, and their
// images), small enough that three CTAs of eight warps keep 196 KB of copies
// in flight per SM, and all index work is per warp: the tile's two bases come
// from two ballots each, the element offsets from constants.  The reversal of
// 30 positions takes 24.1 ms with one 2^12-element pair per CTA and per-element
// deposits over every bit, and 6.7 ms here (34.4 GB, 5.1 TB/s, 0.79 of the measured copy
// rate).

constexpr uint32_t kPermBits = 8;  // largest |L|
constexpr uint32_t kPermWarps = 8;

struct PermParams {
  uint32_t m;              // |L|
  uint32_t n;
  uint64_t lane_d[5];      // position bits of lane bit b (0 past m)
  uint64_t di[8];          // position offset of element 32 i
  uint32_t lane_t[5];      // tau_L image of element bit b
  uint32_t ti[8];          // tau_L image of element 32 i
  uint8_t tau[64];         // tau on all positions
  uint8_t from[64];        // tile-index bit deposited at each position (63: none)
};

__device__ __forceinline__ uint32_t perm_slot(uint32_t e) { return e ^ ((e >> 5) & 7u); }

__global__ void __launch_bounds__(32 * kPermWarps)
    k_permute_pairs(double2* __restrict__ state, const __grid_constant__ PermParams P, uint64_t tiles) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  double2* A = reinterpret_cast<double2*>(smraw) + (warp << (kPermBits + 1));
  double2* B = A + (1u << kPermBits);
  const uint32_t cnt = 1u << P.m;
  uint64_t dl = 0;
  uint32_t tl = 0;
#pragma unroll
  for (uint32_t b = 0; b < 5; ++b)
    if ((lane >> b) & 1u) {
      dl |= P.lane_d[b];
      tl |= P.lane_t[b];
    }
  const uint32_t f0 = P.from[lane], f1 = P.from[lane + 32], t0 = P.tau[lane], t1 = P.tau[lane + 32];
  const uint64_t step = (uint64_t)gridDim.x * kPermWarps;
  for (uint64_t t = (uint64_t)blockIdx.x * kPermWarps + warp; t < tiles; t += step) {
    const uint64_t bT = (uint64_t)__ballot_sync(0xffffffffu, (t >> f0) & 1ULL) |
                        ((uint64_t)__ballot_sync(0xffffffffu, (t >> f1) & 1ULL) << 32);
    const uint64_t bU = (uint64_t)__ballot_sync(0xffffffffu, (bT >> t0) & 1ULL) |
                        ((uint64_t)__ballot_sync(0xffffffffu, (bT >> t1) & 1ULL) << 32);
    if (bU < bT) continue;  // tile tau(T) handles this pair
    const bool self = (bU == bT);
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
      const uint32_t e = lane + 32 * i;
      if (e >= cnt) break;
      cp_async16(&A[perm_slot(e)], state + (bT | P.di[i] | dl));
      if (!self) cp_async16(&B[perm_slot(e)], state + (bU | P.di[i] | dl));
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncwarp();
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
      const uint32_t e = lane + 32 * i;
      if (e >= cnt) break;
      // element e of tile U receives element tau_L(e) of tile T
      const uint32_t te = perm_slot(P.ti[i] | tl);
      state[bU | P.di[i] | dl] = A[te];
      if (!self) state[bT | P.di[i] | dl] = B[te];
    }
    __syncwarp();
  }
}

// =========================================================================
// host side: planner
// =========================================================================

inline hc conj(hc a) { return hc{a.re, -a.im}; }
inline bool is_one_hc(hc a) { return a.re == 1.0 && a.im == 0.0; }
inline bool is_unit_phase(hc a) { return fabs(a.re * a.re + a.im * a.im - 1.0) < 1e-12; }

enum PKind { PG_DIAG, PG_U1, PG_U1X, PG_U2 };

struct PGate {
  PKind kind = PG_DIAG;
  uint32_t t0 = 0, t1 = 0;  // physical targets (U2: t0 = MSB of the gate index)
  uint64_t ctrl = 0;        // physical controls (all must be 1)
  hc u[16];
  bool real = false;
  bool had = false;         // uncontrolled s*[[1,1],[1,-1]]: add/sub, scale deferred
  // diagonal terms
  hc cst{1, 0};
  int nlin = 0;
  uint32_t lq[2] = {0, 0};
  hc lw[2];
  bool quad = false;
  uint32_t qa = 0, qb = 0;
  hc qw{1, 0};
  uint64_t touched = 0;
};

// Extended-precision complex numbers of the rotation planner: the phases and
// divided-out cosines of hundreds of gates multiply up on the host, and are
// rounded to double once, in the tables the kernel reads.
struct hx {
  long double re, im;
};
inline hx operator*(hx a, hx b) { return hx{a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }
inline hx conj(hx a) { return hx{a.re, -a.im}; }
inline bool is_one_hc(hx a) { return a.re == 1.0L && a.im == 0.0L; }
inline hc rounded(hx a) { return hc{(double)a.re, (double)a.im}; }
// A diagonal entry (rounded to double) as a factor of a polynomial.  X and CX
// turn factors into their inverses, taken as conjugates: they have to be of
// modulus one beyond double (or the 2-norm drifts with every such turn).  What
// is divided out goes to *m, to the power of the share of the amplitudes that
// the factor acts on.
inline void factor_of(hc z, int, hc* out, long double*) { *out = z; }
inline void factor_of(hc z, int halves, hx* out, long double* m) {
  const long double a = z.re, b = z.im;
  long double r = sqrtl(a * a + b * b);
  *out = hx{a / r, b / r};
  for (; halves > 0; --halves) r = sqrtl(r);
  *m *= r;
}

template <class C>
struct PolyT {
  uint32_t n = 0;
  std::vector<C> lin;
  std::vector<char> hl;
  std::vector<C> quad;
  std::vector<char> hq;
  std::vector<int> cnt;
  C cst{1, 0};
  bool has_cst = false;

  void init(uint32_t nq) {
    n = nq;
    lin.assign(n, C{1, 0});
    hl.assign(n, 0);
    quad.assign((size_t)n * n, C{1, 0});
    hq.assign((size_t)n * n, 0);
    cnt.assign(n, 0);
    cst = C{1, 0};
    has_cst = false;
  }
  void mul_lin(uint32_t q, C w) {
    if (!hl[q]) { hl[q] = 1; ++cnt[q]; lin[q] = w; } else lin[q] = lin[q] * w;
  }
  void mul_quad(uint32_t a, uint32_t b, C w) {
    const uint32_t lo = std::min(a, b), hi = std::max(a, b);
    const size_t k = (size_t)lo * n + hi;
    if (!hq[k]) { hq[k] = 1; ++cnt[lo]; ++cnt[hi]; quad[k] = w; } else quad[k] = quad[k] * w;
  }
  void add(const PGate& g) {
    long double m = 1.0L;  // the gate's rounding of the norm
    auto up = [&](hc z, int halves) {
      C w;
      factor_of(z, halves, &w, &m);
      return w;
    };
    if (!(g.cst.re == 1.0 && g.cst.im == 0.0)) { cst = cst * up(g.cst, 0); has_cst = true; }
    for (int i = 0; i < g.nlin; ++i) mul_lin(g.lq[i], up(g.lw[i], 1));
    if (g.quad) mul_quad(g.qa, g.qb, up(g.qw, 2));
    if (m != 1.0L) {
      cst.re *= m;
      cst.im *= m;
      has_cst = true;
    }
  }
  bool has_quad(uint32_t a, uint32_t b) const {
    return hq[(size_t)std::min(a, b) * n + std::max(a, b)] != 0;
  }
  // The terms after an X on t: x_t -> 1 - x_t.
  void through_x(uint32_t t) {
    if (hl[t]) {
      cst = cst * lin[t];
      has_cst = true;
      lin[t] = conj(lin[t]);
    }
    for (uint32_t r = 0; r < n; ++r) {
      if (r == t || !has_quad(t, r)) continue;
      C& v = quad[(size_t)std::min(t, r) * n + std::max(t, r)];
      mul_lin(r, v);
      v = conj(v);
    }
  }
  // The terms after a CX: x_t -> x_t + x_c - 2 x_t x_c.  Second degree only
  // when no term pairs t with a third qubit (false: nothing done).
  bool through_cx(uint32_t c, uint32_t t) {
    const bool own = has_quad(c, t);
    if (cnt[t] - (hl[t] ? 1 : 0) - (own ? 1 : 0) > 0) return false;
    const C w = hl[t] ? lin[t] : C{1, 0};
    const size_t k = (size_t)std::min(c, t) * n + std::max(c, t);
    const C v = own ? quad[k] : C{1, 0};
    if (!hl[t] && !own) return true;
    mul_lin(c, w * v);
    const C nq = conj(w) * conj(w) * conj(v);
    if (own) quad[k] = nq;
    else mul_quad(c, t, nq);
    return true;
  }
  bool pending(uint32_t q) const { return cnt[q] > 0; }
  bool empty() const {
    for (uint32_t q = 0; q < n; ++q)
      if (cnt[q]) return false;
    return true;
  }
  // remove and return all terms containing q
  void take(uint32_t q, C* wlin, std::vector<std::pair<uint32_t, C>>& partners) {
    *wlin = hl[q] ? lin[q] : C{1, 0};
    if (hl[q]) { hl[q] = 0; --cnt[q]; lin[q] = C{1, 0}; }
    partners.clear();
    for (uint32_t r = 0; r < n; ++r) {
      if (r == q) continue;
      const uint32_t lo = std::min(q, r), hi = std::max(q, r);
      const size_t k = (size_t)lo * n + hi;
      if (!hq[k]) continue;
      partners.push_back({r, quad[k]});
      hq[k] = 0;
      quad[k] = C{1, 0};
      --cnt[q];
      --cnt[r];
    }
  }
};
using Poly = PolyT<hc>;
using PolyX = PolyT<hx>;

struct POp {
  uint32_t type;
  int gate = -1;            // index into the segment's gate list
  uint32_t q = 0;           // FLUSH target (physical)
  hc wlin{1, 0};
  std::vector<std::pair<uint32_t, hc>> partners;   // FLUSH partners (physical)
  hc gcst{1, 0};                                  // GPHASE constant
  std::vector<std::pair<uint64_t, hc>> gterms;     // GPHASE per-tile terms (masks)
};

// A rotation phase (dq_sweep.cuh) before it is encoded.
struct MFactor {            // diag(1, w) on q, times pr.second for every set partner qubit
  uint32_t q = ~0u;         // ~0: a factor of the whole tile (w and terms)
  hx w{1, 0};
  std::vector<std::pair<uint32_t, hx>> partners;
  std::vector<std::pair<uint64_t, hx>> terms;
};
struct MPhase {
  std::vector<uint32_t> regs;      // physical, RB of them; the rotated ones first
  std::vector<double> t;           // rotations on regs[0..]
  std::vector<std::pair<uint32_t, uint32_t>> flips;  // (control outside the tile, register qubit)
  bool table = false;              // product of cst, lin and quad over the register qubits
  hx cst{1, 0}, lin[4], quad[4][4];
  std::vector<MFactor> cross;      // of register qubits
  std::vector<MFactor> fin;        // final flush
  uint32_t vec[kMaxM];             // address vector of every local bit, and the common offset
  uint32_t off = 0;
};

struct PSweep {
  std::vector<uint32_t> local;  // physical, ascending, size m
  std::vector<POp> ops;
  std::vector<MPhase> micro;    // rotation phases (then ops is empty)
  size_t bytes = 0;             // what their program takes at most, and its slots
  uint32_t slots = 0;
};

// Blob writer (16-byte aligned sections)
struct Blob {
  std::vector<uint8_t> buf;
  size_t align16() {
    while (buf.size() % 16) buf.push_back(0);
    return buf.size();
  }
  template <class T>
  size_t put(const T* p, size_t count) {
    const size_t off = align16();
    const uint8_t* s = reinterpret_cast<const uint8_t*>(p);
    buf.insert(buf.end(), s, s + sizeof(T) * count);
    return off;
  }
};

struct Planner {
  uint32_t n = 0, M = 12, RB = 5, TB = 8;
  // FP64 work per amplitude one sweep may take on: at 30 qubits a sweep's
  // compute stays cheaper than another pass over the state up to ~100
  // (brickwork28 of u3 + cx: 255 ms at 48, 227 ms at 96, the same above)
  double budget = 96.0;
  uint32_t max_ops = 40;    // non-diagonal gates per sweep (bounds the staged program)
  bool single_tile = false;
  // qubits every tile holds (0..4: 512-byte runs; 0..2: 128-byte runs)
  uint64_t pinned = 0x1FULL;
  bool pin_auto = false;
  bool micro_ok = false;  // the launches of this geometry have the micro build

  // cost in FP64 instructions per amplitude
  double gate_cost(const PGate& g) const {
    const double frac = 1.0 / (double)(1ULL << __builtin_popcountll(g.ctrl));
    switch (g.kind) {
      case PG_U1: return g.had ? 2.0 : (g.real ? 4.0 : 8.0) * frac;
      case PG_U1X: return 0.5;
      case PG_U2: return 16.0 * frac;
      default: return 0.0;
    }
  }

  static uint64_t targets(const PGate& g) {
    if (g.kind == PG_DIAG) return 0;
    if (g.kind == PG_U2) return (1ULL << g.t0) | (1ULL << g.t1);
    return 1ULL << g.t0;
  }

  // Split the gate list into sweeps; poly carries pending diagonal terms.
  void plan(std::vector<PGate>& G, Poly& poly, std::vector<PSweep>& out) {
    std::vector<int> rem(G.size());
    for (size_t i = 0; i < G.size(); ++i) rem[i] = (int)i;
    const uint64_t low_mask = single_tile ? ((n >= 64) ? ~0ULL : ((1ULL << n) - 1)) : pinned;
    while (!rem.empty()) {
      uint64_t S = low_mask;
      uint64_t blocked = 0;
      double cost = 0.0;
      std::vector<int> incl, next;
      bool any_nd = false;
      uint32_t nd_count = 0;
      uint64_t diag_touched = 0;
      // conservative size of the encoded program: op + matrix, and a flush
      // per target (op, lane/warp/register tables, slot and its non-local terms)
      size_t bytes = 4096 + 3072;
      const size_t flush_bytes = 48 + 16 * (32 + 8 + 16) + 32 + 32 * (size_t)n;
      for (int gi : rem) {
        const PGate& g = G[gi];
        if (g.touched & blocked) {
          next.push_back(gi);
          blocked |= g.touched;
          continue;
        }
        if (g.kind == PG_DIAG) {
          incl.push_back(gi);
          diag_touched |= g.touched;
          continue;
        }
        const uint64_t need = targets(g);
        const uint64_t ns = S | need;
        double c = gate_cost(g);
        uint64_t tm = need;
        while (tm) {
          const int t = __builtin_ctzll(tm);
          tm &= tm - 1;
          if (poly.pending((uint32_t)t) || ((diag_touched >> t) & 1ULL)) c += 4.0;  // a flush
        }
        const size_t gb = 48 + 16 * 16 + flush_bytes * (size_t)__builtin_popcountll(need);
        const bool fits = (uint32_t)__builtin_popcountll(ns) <= M && nd_count < max_ops &&
                          bytes + gb <= (size_t)max_prog((int)M) - 8192;
        const bool afford = single_tile || !any_nd || cost + c <= budget;
        if (!fits || !afford) {
          next.push_back(gi);
          blocked |= g.touched;
          continue;
        }
        S = ns;
        cost += c;
        bytes += gb;
        any_nd = true;
        ++nd_count;
        incl.push_back(gi);
      }
      // pad the local set to M qubits now: every later decision (which flush
      // partners are local, which per-tile terms test base bits) depends on it
      for (uint32_t q = 0; q < n && (uint32_t)__builtin_popcountll(S) < M; ++q) S |= 1ULL << q;
      PSweep sw;
      for (int gi : incl) {
        const PGate& g = G[gi];
        if (g.kind == PG_DIAG) {
          poly.add(g);
          continue;
        }
        uint64_t tm = targets(g);
        while (tm) {
          const uint32_t t = (uint32_t)__builtin_ctzll(tm);
          tm &= tm - 1;
          if (poly.pending(t)) {
            POp f;
            f.type = OP_FLUSH_R;
            f.q = t;
            poly.take(t, &f.wlin, f.partners);
            sw.ops.push_back(std::move(f));
          }
        }
        POp op;
        op.type = g.kind == PG_U1 ? (g.had ? OP_U1H : g.real ? OP_U1R : OP_U1)
                  : g.kind == PG_U1X ? OP_U1X : OP_U2;
        op.gate = gi;
        sw.ops.push_back(std::move(op));
      }
      for (uint32_t q = 0; q < n; ++q)
        if (S >> q & 1ULL) sw.local.push_back(q);
      out.push_back(std::move(sw));
      rem.swap(next);
    }
  }

  // Apply every pending term in the last sweep (appending one if needed).
  void final_flush(Poly& poly, std::vector<PSweep>& sweeps) {
    if (poly.empty() && !poly.has_cst) return;
    if (sweeps.empty()) {
      PSweep sw;
      uint64_t S = single_tile ? ((n >= 64) ? ~0ULL : ((1ULL << n) - 1)) : pinned;
      for (uint32_t q = 0; q < n && (uint32_t)__builtin_popcountll(S) < M; ++q)
        if (poly.pending(q)) S |= 1ULL << q;
      for (uint32_t q = 0; q < n && (uint32_t)__builtin_popcountll(S) < M; ++q) S |= 1ULL << q;
      for (uint32_t q = 0; q < n; ++q)
        if (S >> q & 1ULL) sw.local.push_back(q);
      sweeps.push_back(std::move(sw));
    }
    PSweep& last = sweeps.back();
    uint64_t S = 0;
    for (uint32_t q : last.local) S |= 1ULL << q;
    for (uint32_t q = 0; q < n; ++q) {
      if (!(S >> q & 1ULL) || !poly.pending(q)) continue;
      POp f;
      f.type = OP_FLUSH_T;  // resolved to R/T by the phase layout
      f.q = q;
      poly.take(q, &f.wlin, f.partners);
      last.ops.push_back(std::move(f));
    }
    // what is left involves non-local qubits only: a per-tile constant
    POp gp;
    gp.type = OP_GPHASE;
    gp.gcst = poly.has_cst ? poly.cst : hc{1, 0};
    for (uint32_t q = 0; q < n; ++q) {
      if (poly.hl[q]) gp.gterms.push_back({1ULL << q, poly.lin[q]});
      for (uint32_t r = q + 1; r < n; ++r) {
        const size_t k = (size_t)q * n + r;
        if (poly.hq[k]) gp.gterms.push_back({(1ULL << q) | (1ULL << r), poly.quad[k]});
      }
    }
    const bool trivial = gp.gterms.empty() && gp.gcst.re == 1.0 && gp.gcst.im == 0.0;
    if (!trivial) last.ops.push_back(std::move(gp));
    poly.init(n);
  }
};

// ---- rotation phases: one-qubit gates as phases and real rotations ----------------------
//
// Host arithmetic is in extended precision, so rounding is the kernel's alone:
// against an 80-bit simulation, 40 layers of 13-qubit brickwork are off by
// 4.3-6.2e-15 (2-norm; 4.6-6.3e-15 with the gates applied as complex 2x2s), and
// 8 layers of rx or ry, rz and rzz on 14 qubits by 1.9e-15 (2.2e-15).

// The segment is made of one-qubit gates, X / CX and diagonal gates, with at
// least one gate that is neither diagonal nor real: real and Hadamard-only
// segments have straight-line builds of their own.
bool micro_eligible(const std::vector<PGate>& G) {
  bool general = false;
  for (const PGate& g : G) {
    if (g.kind == PG_U2 || (g.kind == PG_U1 && g.ctrl != 0)) return false;
    if (g.kind == PG_U1X && __builtin_popcountll(g.ctrl) > 1) return false;
    if (g.kind == PG_U1 && !g.real) general = true;
  }
  return general;
}

// u = r cst diag(1, phi) [[c, -s], [s, c]] diag(1, lam) with real r, c, s >= 0
// and unit phi, lam (cst comes back with r); false when u is not unitary to
// rounding.  u's entries are rounded one by one, so this is the least-squares
// fit: the state then follows the rounded gates, their common loss or gain of
// norm (r) included, and differs from gate by gate arithmetic by little more
// than the rounding of either.
bool split_unitary(const hc* u, long double* c, long double* s, hx* cst, hx* phi, hx* lam) {
  auto up = [](hc z) { return hx{z.re, z.im}; };
  auto mod = [](hx z) { return sqrtl(z.re * z.re + z.im * z.im); };
  auto unit = [&](hx z) {
    const long double r = mod(z);
    return hx{z.re / r, z.im / r};
  };
  const long double m0 = mod(up(u[0])), m1 = mod(up(u[1])), m2 = mod(up(u[2])), m3 = mod(up(u[3]));
  const long double cc = m0 * m0 + m3 * m3, ss = m1 * m1 + m2 * m2, r = sqrtl((cc + ss) / 2.0L);
  if (!(r > 0.0L)) return false;
  *c = sqrtl(cc / 2.0L) / r;
  *s = sqrtl(ss / 2.0L) / r;
  // phases of the diagonal (a) and off-diagonal (b) entries; a0 a3 = b1 b2
  const bool da = m0 > 0.0L && m3 > 0.0L, db = m1 > 0.0L && m2 > 0.0L;
  if (!da && !db) return false;
  hx a0{1, 0}, a3{1, 0}, b1{1, 0}, b2{1, 0};
  if (da) {
    a0 = unit(up(u[0]));
    a3 = unit(up(u[3]));
  }
  if (db) {
    b1 = unit(up(u[2]));
    b2 = unit(hx{-u[1].re, -u[1].im});
  }
  if (!da) a3 = b1 * b2;
  if (!db) {
    b1 = a0;
    b2 = a3;
  }
  // what a0 a3 conj(b1 b2) is off one by rounding, shared out by weight
  const hx w = a0 * a3 * conj(b1) * conj(b2);
  auto turn = [&](hx z, long double e) { return unit(hx{z.re - e * z.im, z.im + e * z.re}); };
  const long double ea = -w.im * *s * *s / 2.0L, eb = w.im * *c * *c / 2.0L;
  a0 = turn(a0, ea);
  b1 = turn(b1, eb);
  b2 = turn(b2, eb);
  *phi = b1 * conj(a0);
  *lam = b2 * conj(a0);
  *cst = a0 * hx{r, 0};
  auto off = [&](hc z, hx w) { return mod(hx{z.re - w.re, z.im - w.im}); };
  const hx ms{-*s, 0}, pc{*c, 0}, ps{*s, 0};
  return fabsl(r - 1.0L) < 1e-14L && off(u[0], *cst * pc) < 4e-15L && off(u[1], *cst * *lam * ms) < 4e-15L &&
         off(u[2], *cst * *phi * ps) < 4e-15L && off(u[3], *cst * *phi * *lam * pc) < 4e-15L;
}

// The banks (of 16 bytes) that sums of address vectors reach.
struct BankSpan {
  uint32_t have = 1;  // bit v: the bank offset v is a sum of the vectors added
  bool add(uint32_t vec) {
    const uint32_t v = vec & 7u;
    if (have >> v & 1u) return false;
    uint32_t more = have;
    for (uint32_t u = 0; u < 8; ++u)
      if (have >> u & 1u) more |= 1u << (u ^ v);
    have = more;
    return true;
  }
  bool all() const { return have == 0xffu; }
};

struct MicroPlanner {
  const Planner& pl;
  // Against Planner::budget (96): a sweep takes up to 60 rotations.  28-qubit
  // brickwork of 20 layers: 105 ms, 108 ms with up to 42, 110 ms with up to 29.
  // X and CX cost nothing here; where they need phases, the program's size ends
  // the sweep (full).
  static constexpr double rot_cost = 1.6;
  static constexpr uint32_t max_rot = 64;
  // The segment with general gates split into phase, rotation (|t| <= 1) and
  // phase: small records, since every sweep and phase scans them.
  struct MGate {
    uint64_t touched;
    PKind kind;                          // PG_DIAG, PG_U1 (a rotation) or PG_U1X
    uint32_t t0;
    int ctrl;                            // PG_U1X: control qubit or -1
    int src;                             // PG_DIAG: the segment's gate, or -1: cst diag(1, w) on t0
    double t;                            // the rotation [[1, -t], [t, 1]] / sqrt(1 + t^2)
    hx w, cst;
  };
  std::vector<MGate> G;
  const std::vector<PGate>* in = nullptr;
  bool ok = true;                        // every gate could be split

  void split(const std::vector<PGate>& gates) {
    in = &gates;
    G.reserve(gates.size() * 4);
    auto diag = [&](uint32_t q, hx w, hx cst) {
      if (is_one_hc(w) && is_one_hc(cst)) return;
      G.push_back(MGate{1ULL << q, PG_DIAG, q, -1, -1, 0.0, w, cst});
    };
    for (size_t i = 0; i < gates.size(); ++i) {
      const PGate& g = gates[i];
      if (g.kind != PG_U1) {
        G.push_back(MGate{g.touched, g.kind, g.t0, g.ctrl ? __builtin_ctzll(g.ctrl) : -1, (int)i, 0.0, hx{1, 0},
                          hx{1, 0}});
        continue;
      }
      long double c, s;
      hx cst, phi, lam;
      if (!split_unitary(g.u, &c, &s, &cst, &phi, &lam)) {
        ok = false;
        return;
      }
      if (c < s) {
        // [[c, -s], [s, c]] = [[s, c], [-c, s]] X Z: the quarter turn costs nothing
        diag(g.t0, lam * hx{-1, 0}, hx{1, 0});
        G.push_back(MGate{g.touched, PG_U1X, g.t0, -1, -1, 0.0, hx{1, 0}, hx{1, 0}});
        const long double x = c;
        c = s;
        s = -x;
      } else {
        diag(g.t0, lam, hx{1, 0});
      }
      const double t = (double)(s / c);
      if (t != 0.0) G.push_back(MGate{g.touched, PG_U1, g.t0, -1, -1, t, hx{1, 0}, hx{1, 0}});
      diag(g.t0, phi, cst);
    }
  }
  void add_diag(PolyX& poly, const MGate& g) const {
    if (g.src >= 0) {
      poly.add((*in)[g.src]);
      return;
    }
    if (!is_one_hc(g.cst)) {
      poly.cst = poly.cst * g.cst;
      poly.has_cst = true;
    }
    if (!is_one_hc(g.w)) poly.mul_lin(g.t0, g.w);
  }

  // Every pending term among the phase's registers, and the constant, as one table.
  void table(MPhase& ph, PolyX& poly) {
    ph.cst = ph.cst * (poly.has_cst ? poly.cst : hx{1, 0});
    ph.table = ph.table || !is_one_hc(ph.cst);
    poly.cst = hx{1, 0};
    poly.has_cst = false;
    for (uint32_t a = 0; a < 4; ++a) {
      const uint32_t x = ph.regs[a];
      ph.lin[a] = hx{1, 0};
      if (poly.hl[x]) {
        ph.table = true;
        ph.lin[a] = poly.lin[x];
        poly.hl[x] = 0;
        --poly.cnt[x];
        poly.lin[x] = hx{1, 0};
      }
      for (uint32_t b = a + 1; b < 4; ++b) {
        const uint32_t y = ph.regs[b];
        ph.quad[a][b] = hx{1, 0};
        if (!poly.has_quad(x, y)) continue;
        const size_t k = (size_t)std::min(x, y) * poly.n + std::max(x, y);
        ph.table = true;
        ph.quad[a][b] = poly.quad[k];
        poly.hq[k] = 0;
        poly.quad[k] = hx{1, 0};
        --poly.cnt[x];
        --poly.cnt[y];
      }
    }
  }
  void take_factor(std::vector<MFactor>& to, PolyX& poly, uint32_t q) {
    MFactor f;
    f.q = q;
    poly.take(q, &f.w, f.partners);
    to.push_back(std::move(f));
  }

  // What the encoded program takes: without phases, of a phase without factors
  // (with its table), of a factor (its slot, a term per qubit or pair outside the
  // tile, its tables).
  size_t frame_bytes() const {
    return sizeof(SwHeader) + sizeof(SwGStore) + ((sizeof(uint64_t) + sizeof(uint32_t)) << (pl.M - kMinRunBits)) +
           16 * 16;  // sections start at multiples of 16
  }
  static size_t factor_bytes(size_t terms, bool tables) {
    return sizeof(SwSlot) + sizeof(SwFinal) + sizeof(SwSlotEnt) * terms + (tables ? sizeof(double2) * (32 + 8 + 16) : 0);
  }
  static constexpr size_t table_bytes = sizeof(double2) * 16;
  static constexpr size_t phase_bytes = sizeof(SwPhase) + sizeof(SwMPhase) + table_bytes;
  void count(PSweep& sw, const MPhase& ph) const {
    sw.bytes += phase_bytes - (ph.table ? 0 : table_bytes);
    for (const auto* fs : {&ph.cross, &ph.fin})
      for (const MFactor& f : *fs) {
        sw.bytes += factor_bytes(f.terms.size() + f.partners.size(), !f.partners.empty());
        ++sw.slots;
      }
  }
  // No room for a phase with four factors and the phase that may close the sweep.
  bool full(const PSweep& sw) const {
    return sw.bytes + 2 * phase_bytes + 4 * factor_bytes(pl.n, true) > (size_t)max_prog((int)pl.M) ||
           sw.slots + 4 > (uint32_t)kMaxSlots;
  }

  struct Tile {            // addresses of the local qubits (of the tile being planned)
    uint64_t S = 0, all = 0;  // local qubits; qubits its gates touch
    int lidx[64];
    uint32_t vec[kMaxM], off = 0;
  };
  void seal(MPhase& ph, const Tile& T) {
    memcpy(ph.vec, T.vec, sizeof(ph.vec));
    ph.off = T.off;
  }
  // Fills the phase's registers with the highest local qubits that are left, so
  // that qubits 0..2 stay thread bits.  vec (null for a phase that writes the
  // state, whose thread order is fixed): those first that leave thread bits
  // reaching every bank.
  void fill(MPhase& ph, const std::vector<uint32_t>& local, const uint32_t* vec) {
    auto has = [&](uint32_t q) { return std::find(ph.regs.begin(), ph.regs.end(), q) != ph.regs.end(); };
    for (size_t k = local.size(); vec && k-- > 0 && ph.regs.size() < 4;) {
      if (has(local[k])) continue;
      BankSpan left;
      for (size_t i = 0; i < local.size(); ++i)
        if (i != k && !has(local[i])) left.add(vec[i]);
      if (left.all()) ph.regs.push_back(local[k]);
    }
    for (size_t k = local.size(); k-- > 0 && ph.regs.size() < 4;)
      if (!has(local[k])) ph.regs.push_back(local[k]);
  }

  // The phases of the gates `todo` (program order), whose targets are in the
  // tile.  Returns those that a full sweep has no room for.
  std::vector<int> phases(std::vector<int> todo, PSweep& sw, PolyX& poly) {
    Tile T;
    sw.bytes = frame_bytes();
    for (int& x : T.lidx) x = -1;
    for (int gi : todo) T.all |= G[gi].touched;
    for (uint32_t k = 0; k < sw.local.size(); ++k) {
      T.S |= 1ULL << sw.local[k];
      T.lidx[sw.local[k]] = (int)k;
      T.vec[k] = swz(1u << k);
    }
    // Runs f(gate) over the gates in order; those it takes (true) are removed,
    // a gate behind one that stays on a shared qubit is not offered.
    auto scan = [&](auto f) {
      uint64_t blocked = 0;
      size_t stay = 0;
      for (size_t i = 0; i < todo.size(); ++i) {
        const MGate& g = G[todo[i]];
        if (!(g.touched & blocked) && f(g)) continue;
        todo[stay++] = todo[i];
        blocked |= g.touched;
        if (blocked == T.all) {  // nothing later can be offered
          for (++i; i < todo.size(); ++i) todo[stay++] = todo[i];
          break;
        }
      }
      const bool any = stay != todo.size();
      todo.resize(stay);
      return any;
    };
    auto diagonal = [&](const MGate& g) {
      if (g.kind != PG_DIAG) return false;
      add_diag(poly, g);
      return true;
    };
    while (!todo.empty()) {
      // what executes nothing: diagonal gates, X, and CX inside the tile
      uint64_t must = 0;  // targets whose pending terms a CX cannot pass
      while (scan([&](const MGate& g) -> bool {
        if (diagonal(g)) return true;
        if (g.kind != PG_U1X) return false;
        const uint32_t vt = T.vec[T.lidx[g.t0]];
        if (g.ctrl < 0) {
          poly.through_x(g.t0);
          T.off ^= vt;
          return true;
        }
        const uint32_t c = (uint32_t)g.ctrl;
        if (T.lidx[c] < 0) return false;
        if (!poly.through_cx(c, g.t0)) {
          must |= 1ULL << g.t0;
          return false;
        }
        T.vec[T.lidx[c]] ^= vt;
        return true;
      })) {
      }
      if (todo.empty() || full(sw)) break;
      // targets that can go into a phase now, in program order
      std::vector<uint32_t> cand;
      uint64_t seen = 0, blocked = 0;
      for (int gi : todo) {
        const MGate& g = G[gi];
        const bool now = g.kind != PG_DIAG && !(g.touched & blocked);
        if (now && !((seen >> g.t0) & 1ULL)) {
          cand.push_back(g.t0);
          seen |= 1ULL << g.t0;
        }
        // (a control outside the tile is no one's target here)
        blocked |= now && g.ctrl >= 0 && T.lidx[g.ctrl] < 0 ? 1ULL << g.t0 : g.touched;
      }
      // up to four of them, a target's quadratic partners with it; spare places
      // to partners that are not targets now (their terms then need no factor
      // of their own)
      std::vector<uint32_t> pick;
      auto has = [](const std::vector<uint32_t>& v, uint32_t q) { return std::find(v.begin(), v.end(), q) != v.end(); };
      auto add_partners = [&](uint32_t q, bool targets) {
        for (uint32_t r = 0; r < poly.n && pick.size() < 4; ++r)
          if (r != q && poly.has_quad(q, r) && (T.S >> r & 1ULL) && !has(pick, r) && (!targets || (seen >> r & 1ULL)))
            pick.push_back(r);
      };
      for (uint32_t q : cand) {
        if (pick.size() >= 4) break;
        if (has(pick, q)) continue;
        pick.push_back(q);
        add_partners(q, true);
      }
      for (size_t i = 0; i < pick.size(); ++i) add_partners(pick[i], false);
      uint64_t R = 0;
      for (uint32_t q : pick) R |= 1ULL << q;
      MPhase ph;
      // X controlled from outside the tile
      scan([&](const MGate& g) {
        if (g.kind != PG_U1X || g.ctrl < 0 || !(R >> g.t0 & 1ULL) || (must >> g.t0 & 1ULL)) return false;
        const uint32_t c = (uint32_t)g.ctrl;
        if (T.lidx[c] >= 0 || ph.flips.size() >= 4) return false;
        if (!poly.through_cx(c, g.t0)) {
          must |= 1ULL << g.t0;
          return false;
        }
        ph.flips.push_back({c, g.t0});
        return true;
      });
      while (scan(diagonal)) {
      }
      // rotations of the picked qubits (not of one whose terms a CX waits for)
      std::vector<int> rots;
      scan([&](const MGate& g) {
        if (g.kind != PG_U1 || !(R >> g.t0 & 1ULL)) return false;
        for (int x : rots)
          if (G[x].t0 == g.t0) return false;
        rots.push_back((int)(&g - G.data()));
        return true;
      });
      for (int x : rots) ph.regs.push_back(G[x].t0);
      for (uint32_t q : pick)
        if (!has(ph.regs, q)) ph.regs.push_back(q);
      fill(ph, sw.local, T.vec);
      table(ph, poly);
      for (uint32_t q : ph.regs)
        if (poly.pending(q) && (must >> q & 1ULL || std::any_of(rots.begin(), rots.end(), [&](int x) {
              return G[x].t0 == q;
            })))
          take_factor(ph.cross, poly, q);
      for (int x : rots) {
        const double t = G[x].t;
        ph.t.push_back(t);
        poly.cst = poly.cst * hx{1.0L / sqrtl(1.0L + (long double)t * t), 0};  // of the rounded t
        poly.has_cst = true;
      }
      seal(ph, T);
      count(sw, ph);
      sw.micro.push_back(std::move(ph));
    }
    // the last phase writes the state by logical addresses: qubits 0..2 must be
    // its thread bits, and no address change may follow it
    const MPhase* last = sw.micro.empty() ? nullptr : &sw.micro.back();
    bool direct = last && memcmp(last->vec, T.vec, sizeof(uint32_t) * sw.local.size()) == 0 && last->off == T.off;
    if (direct)
      for (uint32_t q : last->regs)
        if (q < 3) direct = false;
    if (!direct) {
      MPhase ph;
      fill(ph, sw.local, nullptr);
      for (auto& x : ph.lin) x = hx{1, 0};
      for (auto& r : ph.quad)
        for (auto& x : r) x = hx{1, 0};
      seal(ph, T);
      count(sw, ph);
      sw.micro.push_back(std::move(ph));
    }
    return todo;
  }

  void plan(PolyX& poly, std::vector<PSweep>& out) {
    std::vector<int> rem(G.size());
    for (size_t i = 0; i < G.size(); ++i) rem[i] = (int)i;
    uint64_t all = 0;
    for (const MGate& g : G) all |= g.touched;
    const uint64_t low = pl.single_tile ? ((1ULL << pl.n) - 1) : pl.pinned;
    while (!rem.empty()) {
      // the gates of this sweep, as in Planner::plan
      uint64_t S = low, blocked = 0;
      double cost = 0.0;
      uint32_t rots = 0;
      bool any = false;
      std::vector<int> incl, next;
      for (size_t i = 0; i < rem.size(); ++i) {
        const int gi = rem[i];
        const MGate& g = G[gi];
        if (blocked == all) {  // nothing later can be taken
          next.insert(next.end(), rem.begin() + (ptrdiff_t)i, rem.end());
          break;
        }
        bool take = !(g.touched & blocked);
        if (take && g.kind != PG_DIAG) {
          const uint64_t ns = S | (1ULL << g.t0);
          const double c = g.kind == PG_U1X ? 0.0 : rot_cost;
          take = (uint32_t)__builtin_popcountll(ns) <= pl.M && (g.kind == PG_U1X || rots < max_rot) &&
                 (!any || cost + c <= pl.budget);
          if (take) {
            S = ns;
            cost += c;
            any = true;
            rots += g.kind != PG_U1X;
          }
        }
        if (take) {
          incl.push_back(gi);
        } else {
          next.push_back(gi);
          blocked |= g.touched;
        }
      }
      for (uint32_t q = 0; q < pl.n && (uint32_t)__builtin_popcountll(S) < pl.M; ++q) S |= 1ULL << q;
      PSweep sw;
      for (uint32_t q = 0; q < pl.n; ++q)
        if (S >> q & 1ULL) sw.local.push_back(q);
      rem.swap(next);
      if (!any) {
        for (int gi : incl) add_diag(poly, G[gi]);
        continue;
      }
      const std::vector<int> left = phases(std::move(incl), sw, poly);
      out.push_back(std::move(sw));
      if (left.empty()) continue;
      next.clear();
      std::merge(rem.begin(), rem.end(), left.begin(), left.end(), std::back_inserter(next));
      rem.swap(next);
    }
  }

  // Every pending term, in a last phase of the last sweep, or where that has no
  // room for it in a sweep of its own (whose program is well below the limit:
  // a factor per tile qubit and a term per pair of qubits).
  void final_flush(PolyX& poly, std::vector<PSweep>& sweeps) {
    if (poly.empty() && !poly.has_cst) return;
    PSweep& last = sweeps.back();
    MPhase ph;
    fill(ph, last.local, nullptr);
    table(ph, poly);
    for (uint32_t q : ph.regs)
      if (poly.pending(q)) take_factor(ph.cross, poly, q);
    for (uint32_t q : last.local)
      if (poly.pending(q)) take_factor(ph.fin, poly, q);
    MFactor tile;
    for (uint32_t q = 0; q < poly.n; ++q) {
      if (poly.hl[q]) tile.terms.push_back({1ULL << q, poly.lin[q]});
      for (uint32_t r = q + 1; r < poly.n; ++r)
        if (poly.has_quad(q, r)) tile.terms.push_back({(1ULL << q) | (1ULL << r), poly.quad[(size_t)q * poly.n + r]});
    }
    if (!tile.terms.empty()) ph.fin.push_back(std::move(tile));
    poly.init(poly.n);
    const size_t used = last.bytes;
    count(last, ph);
    if (last.bytes > (size_t)max_prog((int)pl.M) || last.slots > (uint32_t)kMaxSlots) {
      PSweep own;
      own.local = last.local;
      own.bytes = frame_bytes() + last.bytes - used;
      for (uint32_t k = 0; k < own.local.size(); ++k) ph.vec[k] = swz(1u << k);
      own.micro.push_back(std::move(ph));
      sweeps.push_back(std::move(own));
      return;
    }
    // after an address change (of an empty last phase, or none) the state's order
    const MPhase& before = last.micro.back();
    memcpy(ph.vec, before.vec, sizeof(ph.vec));
    ph.off = before.off;
    // an empty last phase is replaced
    if (before.t.empty() && !before.table && before.cross.empty() && before.flips.empty()) last.micro.pop_back();
    last.micro.push_back(std::move(ph));
  }
};

// Thread-bit order: lanes 0..2 take bits with linearly independent swizzle
// vectors, the first ones there are.  With three of them eight lanes reach all
// banks.  CX gates folded into the address vectors can leave fewer, where a
// phase's own qubits need the rest in registers: its accesses then take two to
// eight times as long, at the right addresses all the same.
void order_thread_bits(std::vector<uint32_t>& tb, const uint32_t* vec) {
  std::vector<uint32_t> lead, rest;
  BankSpan span;
  for (uint32_t b : tb) (span.add(vec[b]) ? lead : rest).push_back(b);
  lead.insert(lead.end(), rest.begin(), rest.end());
  tb = lead;
}

// Thread and register layout of a phase whose register bits are the local
// bits `regs`: address tables, and the places of each local bit.  vec: the
// address vector of every local bit, off: the address of element 0; keep_low:
// local bits 0..2 are lanes 0..2 (a direct write of the state).
struct PhaseLayout {
  std::vector<uint32_t> tb;        // local bits of the thread bits
  int rix[kMaxM], tix[kMaxM];      // register / thread bit of a local bit, or -1
};
int phase_layout(const std::vector<uint32_t>& regs, uint32_t m, uint32_t TBn, uint32_t RB, const uint32_t* vec,
                 uint32_t off, bool keep_low, SwPhase& sp, PhaseLayout& pl) {
  const int kSwTB = (int)TBn;
  pl.tb.clear();
  for (uint32_t b = 0; b < m; ++b)
    if (std::find(regs.begin(), regs.end(), b) == regs.end()) pl.tb.push_back(b);
  if (pl.tb.size() != (size_t)kSwTB) return fail(DQ_ERR_INTERNAL, "phase without its register bits");
  if (!keep_low) order_thread_bits(pl.tb, vec);
  for (int i = 0; i < kMaxM; ++i) pl.rix[i] = pl.tix[i] = -1;
  for (uint32_t b = 0; b < RB; ++b) {
    sp.V[b] = vec[regs[b]];
    pl.rix[regs[b]] = (int)b;
  }
  for (uint32_t b = RB; b < 4; ++b) sp.V[b] = 0;
  for (int i = 0; i < kSwTB; ++i) pl.tix[pl.tb[i]] = i;
  for (uint32_t ln = 0; ln < 32; ++ln) {
    sp.lanesw[ln] = off;
    for (int i = 0; i < 5; ++i)
      if ((ln >> i) & 1u) sp.lanesw[ln] ^= vec[pl.tb[i]];
  }
  for (uint32_t wp = 0; wp < 8; ++wp) {
    sp.warpsw[wp] = 0;
    for (int i = 0; i + 5 < kSwTB; ++i)
      if ((wp >> i) & 1u) sp.warpsw[wp] ^= vec[pl.tb[5 + i]];
  }
  return DQ_OK;
}

// Encode a planned sweep into the device blob format.  general_ops: rotation
// phases are also written in the general op set (plan inspection; no kernel
// needs them).
int encode_sweep(const PSweep& sw_in, const std::vector<PGate>& G, uint32_t TBn, uint32_t RB,
                 Blob& blob, size_t* offset, bool general_ops) {
  const int kSwTB = (int)TBn;
  const uint32_t m = (uint32_t)sw_in.local.size();
  if (m != kSwTB + RB) return fail(DQ_ERR_INTERNAL, "sweep local set size mismatch");
  int lidx[64];
  for (int i = 0; i < 64; ++i) lidx[i] = -1;
  for (uint32_t k = 0; k < m; ++k) lidx[sw_in.local[k]] = (int)k;

  // Uncontrolled X gates on local bits that no earlier op of the sweep
  // involves (as target or control; any flush or global phase stops the scan
  // for good) commute to the front of the sweep and fold into the tile load:
  // element e is stored at the shared-memory slot of e with those bits
  // flipped (the swizzled layout is XOR-linear), so they cost nothing.
  PSweep sw;
  sw.local = sw_in.local;
  uint32_t tile_xload = 0;
  {
    uint64_t involved = 0;
    bool stopped = false;
    for (const POp& op : sw_in.ops) {
      if (!stopped && op.type == OP_U1X && op.gate >= 0 && G[op.gate].ctrl == 0) {
        const uint32_t t = G[op.gate].t0;
        if (!((involved >> t) & 1ULL) && lidx[t] >= 0) {
          tile_xload ^= swz(1u << (uint32_t)lidx[t]);
          continue;
        }
      }
      if (op.type == OP_FLUSH_R || op.type == OP_FLUSH_T || op.type == OP_GPHASE) stopped = true;
      if (op.gate >= 0) involved |= (1ULL << G[op.gate].t0) | G[op.gate].ctrl |
                                    (op.type == OP_U2 ? (1ULL << G[op.gate].t1) : 0ULL);
      sw.ops.push_back(op);
    }
  }

  // phases: consecutive ops whose register needs fit RB register bits
  struct PhaseTmp {
    std::vector<uint32_t> regs;  // local bits
    size_t ob, oe;
  };
  std::vector<PhaseTmp> phases;
  auto need_of = [&](const POp& op, std::vector<uint32_t>& nd) {
    nd.clear();
    if (op.type == OP_U1 || op.type == OP_U1R || op.type == OP_U1X || op.type == OP_U1H) {
      nd.push_back((uint32_t)lidx[G[op.gate].t0]);
    } else if (op.type == OP_U2) {
      nd.push_back((uint32_t)lidx[G[op.gate].t0]);
      nd.push_back((uint32_t)lidx[G[op.gate].t1]);
    } else if (op.type == OP_FLUSH_R) {
      nd.push_back((uint32_t)lidx[op.q]);   // precedes the gate on q: same phase
    }
  };
  {
    size_t i = 0;
    std::vector<uint32_t> nd;
    while (i < sw.ops.size()) {
      PhaseTmp ph;
      ph.ob = i;
      size_t j = i;
      while (j < sw.ops.size()) {
        need_of(sw.ops[j], nd);
        std::vector<uint32_t> u = ph.regs;
        for (uint32_t b : nd)
          if (std::find(u.begin(), u.end(), b) == u.end()) u.push_back(b);
        if (u.size() > RB) break;
        ph.regs = u;
        ++j;
      }
      if (j == i) return fail(DQ_ERR_INTERNAL, "op needs more register bits than a phase has");
      ph.oe = j;
      phases.push_back(ph);
      i = j;
    }
    if (phases.empty()) phases.push_back(PhaseTmp{{}, 0, 0});
  }

  double scale = 1.0;  // product of the deferred Hadamard factors
  struct EncOp {
    uint32_t type = 0, b0 = 0, b1 = 0, creg = 0, ctl_thr = 0, flags = 0, slot = 0, data = 0;
    uint64_t cnl = 0;
  };
  std::vector<SwPhase> P;
  std::vector<EncOp> O;
  std::vector<SwSlot> SL;
  std::vector<SwSlotEnt> SE;
  std::vector<double2> D;
  auto d2 = [](hc z) { return make_double2(z.re, z.im); };
  auto add_slot = [&](hc w0, const std::vector<std::pair<uint64_t, hc>>& ents) -> uint32_t {
    SwSlot s{};
    s.count = (uint32_t)ents.size();
    s.start = (uint32_t)SE.size();
    s.w0 = d2(w0);
    for (auto& e : ents) {
      SwSlotEnt x{};
      x.mask = e.first;
      x.w = d2(e.second);
      SE.push_back(x);
    }
    SL.push_back(s);
    return (uint32_t)SL.size() - 1;
  };

  uint32_t carry_xload = 0;
  std::vector<uint32_t> last_tb, last_regs;  // thread / register bits of the last phase
  uint32_t plain_vec[kMaxM];
  for (uint32_t k = 0; k < (uint32_t)kMaxM; ++k) plain_vec[k] = swz(1u << k);
  std::vector<SwMPhase> MP;     // rotation phases
  std::vector<SwFinal> FN;
  std::vector<double2> DS;      // data of the general ops of such a sweep only (after D)
  std::vector<char> in_ds;      // per op: data counts from the start of DS
  for (const MPhase& ph : sw_in.micro) {
    SwPhase sp{};
    std::vector<uint32_t> regs;
    for (uint32_t q : ph.regs) regs.push_back((uint32_t)lidx[q]);
    PhaseLayout lay;
    const bool last = &ph == &sw_in.micro.back();
    DQ_TRY(phase_layout(regs, m, TBn, RB, ph.vec, ph.off, last, sp, lay));
    SwMPhase mp{};
    sp.op_begin = (uint32_t)O.size();
    auto push = [&](const EncOp& e, bool ds) {
      if (!general_ops) return;
      O.push_back(e);
      in_ds.push_back(ds ? 1 : 0);
    };
    // the 2x2 m on register bit b, in the general op set
    auto push_u1 = [&](uint32_t type, uint32_t b, uint32_t creg, const hc* mm) {
      EncOp e{};
      e.type = type;
      e.b0 = b;
      e.creg = creg;
      e.data = (uint32_t)DS.size();
      if (general_ops)
        for (int i = 0; i < 4; ++i) DS.push_back(d2(mm[i]));
      push(e, true);
    };
    // slot, thread table and (for the final flush) register table of a factor
    auto factors = [&](const MFactor& f, EncOp& so) {
      std::vector<std::pair<uint64_t, hc>> nl;
      for (const auto& x : f.terms) nl.push_back({x.first, rounded(x.second)});
      hx wthr[kMaxTB], wreg[4];
      for (auto& x : wthr) x = hx{1, 0};
      for (auto& x : wreg) x = hx{1, 0};
      bool thr = false;
      for (const auto& pr : f.partners) {
        const int l = lidx[pr.first];
        if (l < 0) {
          nl.push_back({1ULL << pr.first, rounded(pr.second)});
        } else if (lay.rix[l] >= 0) {
          wreg[lay.rix[l]] = wreg[lay.rix[l]] * pr.second;
          so.flags |= FL_REG;
        } else {
          wthr[lay.tix[l]] = wthr[lay.tix[l]] * pr.second;
          thr = true;
        }
      }
      so.slot = add_slot(rounded(f.w), nl);
      so.data = (uint32_t)D.size();
      if (thr) {
        so.flags |= FL_THR;
        for (uint32_t ln = 0; ln < 32; ++ln) {
          hx w{1, 0};
          for (int i = 0; i < 5; ++i)
            if ((ln >> i) & 1u) w = w * wthr[i];
          D.push_back(d2(rounded(w)));
        }
        for (uint32_t wp = 0; wp < 8; ++wp) {
          hx w{1, 0};
          for (int i = 0; i + 5 < kSwTB; ++i)
            if ((wp >> i) & 1u) w = w * wthr[5 + i];
          D.push_back(d2(rounded(w)));
        }
      }
      if (so.flags & FL_REG)
        for (uint32_t j = 0; j < (1u << RB); ++j) {
          hx w{1, 0};
          for (uint32_t b = 0; b < RB; ++b)
            if ((j >> b) & 1u) w = w * wreg[b];
          D.push_back(d2(rounded(w)));
        }
    };
    if (ph.flips.size() > 4 || ph.t.size() > 4) return fail(DQ_ERR_INTERNAL, "rotation phase too large");
    for (const auto& f : ph.flips) {
      mp.cmask[mp.ncond] = 1ULL << f.first;
      mp.cxor[mp.ncond++] = ph.vec[lidx[f.second]];
      EncOp e{};
      e.type = OP_U1X;
      e.b0 = (uint32_t)lay.rix[lidx[f.second]];
      e.cnl = 1ULL << f.first;
      e.data = (uint32_t)DS.size();
      push(e, true);
    }
    mp.mul = ~0u;
    if (ph.table) {
      mp.mul = (uint32_t)D.size();
      for (uint32_t j = 0; j < (1u << RB); ++j) {
        hx f = ph.cst;
        for (uint32_t x = 0; x < RB; ++x) {
          if (!((j >> x) & 1u)) continue;
          f = f * ph.lin[x];
          for (uint32_t y = x + 1; y < RB; ++y)
            if ((j >> y) & 1u) f = f * ph.quad[x][y];
        }
        D.push_back(d2(rounded(f)));
      }
      for (uint32_t x = 0; x < RB; ++x) {
        const hx one = x == 0 ? ph.cst : hx{1, 0};
        const hc lin[4] = {rounded(one), hc{0, 0}, hc{0, 0}, rounded(one * ph.lin[x])};
        push_u1(OP_U1, x, 0, lin);
        for (uint32_t y = x + 1; y < RB; ++y) {
          const hc qd[4] = {hc{1, 0}, hc{0, 0}, hc{0, 0}, rounded(ph.quad[x][y])};
          if (!is_one_hc(ph.quad[x][y])) push_u1(OP_U1, y, 1u << x, qd);
        }
      }
    }
    for (auto& x : mp.cross) x = ~0u;
    for (const MFactor& f : ph.cross) {
      EncOp so{};
      so.type = OP_FLUSH_R;
      so.b0 = (uint32_t)lay.rix[lidx[f.q]];
      factors(f, so);
      if (so.flags & FL_REG) return fail(DQ_ERR_INTERNAL, "register partner left to a cross factor");
      push(so, false);
      mp.cross[so.b0] = so.slot | (so.flags << 16);
      mp.cdata[so.b0] = so.data;
      ++mp.ncross;
    }
    mp.k = (uint32_t)ph.t.size();
    for (uint32_t x = 0; x < mp.k; ++x) {
      mp.t[x] = ph.t[x];
      const hc r[4] = {hc{1, 0}, hc{-ph.t[x], 0}, hc{ph.t[x], 0}, hc{1, 0}};
      push_u1(OP_U1R, x, 0, r);
    }
    if (!ph.fin.empty() && mp.k) return fail(DQ_ERR_INTERNAL, "final flush in a phase with rotations");
    mp.fin0 = (uint32_t)FN.size();
    for (const MFactor& f : ph.fin) {
      EncOp so{};
      const bool tile = f.q == ~0u;
      so.type = tile ? OP_GPHASE : OP_FLUSH_T;
      so.b0 = tile ? 0u : (uint32_t)lay.tix[lidx[f.q]];
      factors(f, so);
      push(so, false);
      FN.push_back(SwFinal{so.slot, so.flags, tile ? ~0u : so.b0, so.data});
    }
    mp.nfin = (uint32_t)FN.size() - mp.fin0;
    sp.op_end = (uint32_t)O.size();
    last_tb = lay.tb;
    last_regs = regs;
    MP.push_back(mp);
    P.push_back(sp);
  }
  if (!sw_in.micro.empty()) phases.clear();
  for (const PhaseTmp& ph : phases) {
    SwPhase sp{};
    // spare register slots take the highest unused local bits, so that the
    // lowest ones (qubits 0..2) stay thread bits: lanes 0..2 then cover
    // 128-byte runs, which the last phase's direct writes need
    std::vector<uint32_t> regs = ph.regs;
    for (uint32_t b = m; b-- > 0 && regs.size() < RB;)
      if (std::find(regs.begin(), regs.end(), b) == regs.end()) regs.push_back(b);
    PhaseLayout lay;
    DQ_TRY(phase_layout(regs, m, TBn, RB, plain_vec, 0, false, sp, lay));
    const std::vector<uint32_t>& tb = lay.tb;
    const int (&rix)[kMaxM] = lay.rix;
    const int (&tix)[kMaxM] = lay.tix;
    sp.op_begin = (uint32_t)O.size();
    // flush of a register target: per-tile slot, thread/register factor tables
    auto encode_flush = [&](const POp& op, EncOp& so) {
      const int l = lidx[op.q];
      std::vector<std::pair<uint64_t, hc>> nl;
      hc wthr[kMaxTB];
      for (int i = 0; i < kSwTB; ++i) wthr[i] = hc{1, 0};
      hc wreg[5];
      for (int i = 0; i < 5; ++i) wreg[i] = hc{1, 0};
      bool hasF = false;
      for (auto& pr : op.partners) {
        const int pl = lidx[pr.first];
        if (pl < 0) {
          nl.push_back({1ULL << pr.first, pr.second});
        } else if (rix[pl] >= 0) {
          wreg[rix[pl]] = wreg[rix[pl]] * pr.second;
          hasF = true;
        } else {
          wthr[tix[pl]] = wthr[tix[pl]] * pr.second;
        }
      }
      so.slot = add_slot(op.wlin, nl);
      const bool reg_target = rix[l] >= 0;
      bool thr = false;
      for (int i = 0; i < kSwTB; ++i)
        if (!(wthr[i].re == 1.0 && wthr[i].im == 0.0)) thr = true;
      if (thr) {
        so.flags |= FL_THR;
        for (uint32_t ln = 0; ln < 32; ++ln) {  // lane factor: thread bits 0..4
          hc f{1, 0};
          for (int i = 0; i < 5; ++i)
            if ((ln >> i) & 1u) f = f * wthr[i];
          D.push_back(d2(f));
        }
        for (uint32_t wp = 0; wp < 8; ++wp) {   // warp factor: thread bits 5..TB-1
          hc f{1, 0};
          for (int i = 0; i + 5 < kSwTB; ++i)
            if ((wp >> i) & 1u) f = f * wthr[5 + i];
          D.push_back(d2(f));
        }
      }
      if (hasF) {
        so.flags |= FL_REG;
        if (reg_target) {
          const uint32_t B = (uint32_t)rix[l];
          for (uint32_t idx = 0; idx < (1u << (RB - 1)); ++idx) {
            const uint32_t j = ((idx >> B) << (B + 1)) | (idx & ((1u << B) - 1));
            hc f{1, 0};
            for (uint32_t b = 0; b < RB; ++b)
              if (b != B && ((j >> b) & 1u)) f = f * wreg[b];
            D.push_back(d2(f));
          }
        } else {
          for (uint32_t j = 0; j < (1u << RB); ++j) {
            hc f{1, 0};
            for (uint32_t b = 0; b < RB; ++b)
              if ((j >> b) & 1u) f = f * wreg[b];
            D.push_back(d2(f));
          }
        }
      }
    };
    auto is_u1_type = [](uint32_t t) {
      return t == OP_U1 || t == OP_U1R || t == OP_U1X || t == OP_U1H;
    };
    // An uncontrolled X on a register bit that no earlier op of the phase
    // involves (as target, control or, conservatively, any flush) commutes to
    // the front of the phase and becomes part of the load: element j is read
    // from the address of j with that bit flipped (the swizzled addresses are
    // XOR-linear).  involved: register bits touched so far in this phase.
    uint32_t involved = 0;
    for (size_t oi = ph.ob; oi < ph.oe; ++oi) {
      const POp& op = sw.ops[oi];
      EncOp so{};
      so.type = op.type;
      // a flush of a register bit right before an uncontrolled one-qubit op on
      // the same qubit travels inside that op (FL_PRE)
      const POp* pre = nullptr;
      if ((op.type == OP_FLUSH_R || op.type == OP_FLUSH_T) && oi + 1 < ph.oe &&
          is_u1_type(sw.ops[oi + 1].type) && G[sw.ops[oi + 1].gate].ctrl == 0 &&
          G[sw.ops[oi + 1].gate].t0 == op.q && rix[lidx[op.q]] >= 0) {
        pre = &op;
        ++oi;
      }
      const POp& cur = sw.ops[oi];
      so.type = cur.type;
      if (!pre && cur.type == OP_U1X && G[cur.gate].ctrl == 0) {
        const uint32_t b = (uint32_t)rix[lidx[G[cur.gate].t0]];
        if (!((involved >> b) & 1u)) {
          sp.xload ^= sp.V[b];
          continue;
        }
      }
      if (pre || cur.type == OP_FLUSH_R || cur.type == OP_FLUSH_T || cur.type == OP_GPHASE)
        involved = ~0u;
      if (is_u1_type(cur.type) || cur.type == OP_U2) {
        const PGate& g = G[cur.gate];
        if (cur.type == OP_U1H) scale = scale * g.u[0].re;
        // controls: register bits, thread bits, non-local
        uint64_t cm = g.ctrl;
        while (cm) {
          const uint32_t c = (uint32_t)__builtin_ctzll(cm);
          cm &= cm - 1;
          const int l = lidx[c];
          if (l < 0) so.cnl |= 1ULL << c;
          else if (rix[l] >= 0) so.creg |= 1u << rix[l];
          else so.ctl_thr |= 1u << tix[l];
        }
        so.data = (uint32_t)D.size();
        if (cur.type == OP_U2) {
          int r0 = rix[lidx[g.t0]], r1 = rix[lidx[g.t1]];
          hc mm[16];
          for (int i = 0; i < 16; ++i) mm[i] = g.u[i];
          if (r0 > r1) {  // put the lower register bit first: swap the gate's index bits
            const int perm[4] = {0, 2, 1, 3};
            for (int r = 0; r < 4; ++r)
              for (int c = 0; c < 4; ++c) mm[r * 4 + c] = g.u[perm[r] * 4 + perm[c]];
            std::swap(r0, r1);
          }
          so.b0 = (uint32_t)r0;
          so.b1 = (uint32_t)r1;
          for (int i = 0; i < 16; ++i) D.push_back(d2(mm[i]));
        } else {
          so.b0 = (uint32_t)rix[lidx[g.t0]];
          for (int i = 0; i < 4; ++i) D.push_back(d2(g.u[i]));
          if (pre) {
            so.flags |= FL_PRE;
            encode_flush(*pre, so);
          }
        }
      } else if (cur.type == OP_FLUSH_R || cur.type == OP_FLUSH_T) {
        const int l = lidx[cur.q];
        so.data = (uint32_t)D.size();
        encode_flush(cur, so);
        if (rix[l] >= 0) {
          so.type = OP_FLUSH_R;
          so.b0 = (uint32_t)rix[l];
        } else {
          so.type = OP_FLUSH_T;
          so.b0 = (uint32_t)tix[l];
        }
      } else if (cur.type == OP_GPHASE) {
        so.slot = add_slot(cur.gcst, cur.gterms);
      }
      if (is_u1_type(cur.type)) involved |= (1u << so.b0) | so.creg;
      if (cur.type == OP_U2) involved |= (1u << so.b0) | (1u << so.b1) | so.creg;
      O.push_back(so);
    }
    if (&ph == &phases.back() && scale != 1.0) {
      // the deferred 1/sqrt(2) factors: fold into a per-tile phase if there is one
      bool folded = false;
      for (size_t oi = sp.op_begin; oi < O.size(); ++oi)
        if (O[oi].type == OP_GPHASE) {
          SL[O[oi].slot].w0.x *= scale;
          SL[O[oi].slot].w0.y *= scale;
          folded = true;
          break;
        }
      if (!folded) {
        EncOp so{};
        so.type = OP_SCALE;
        so.data = (uint32_t)D.size();
        D.push_back(make_double2(scale, 0.0));
        O.push_back(so);
      }
    }
    // A phase made only of uncontrolled Hadamard-pattern ops on register bits
    // 0, 1, ..., K-1 in that order (register bits are assigned in the order
    // the phase's ops need them), optionally followed by the deferred scale,
    // runs as straight-line code: an OP_HPHASE marker goes in front of them.
    {
      const size_t ob = sp.op_begin, oe = O.size();
      size_t k = 0;
      bool ok = oe > ob, sc = false;
      for (size_t i = ob; i < oe && ok; ++i) {
        const EncOp& x = O[i];
        if (x.type == OP_SCALE && i + 1 == oe && i > ob) {
          sc = true;
          continue;
        }
        ok = (x.type == OP_U1H || x.type == OP_U1R) && x.creg == 0 && x.ctl_thr == 0 && x.cnl == 0 &&
             x.b0 == (uint32_t)k;
        ++k;
      }
      // the deferred scale folds into the last op, which must then be a Hadamard
      if (sc && k >= 1 && O[ob + k - 1].type != OP_U1H) ok = false;
      if (ok && k >= 1 && k <= RB) {
        for (size_t i = ob; i < ob + k; ++i) {
          EncOp& x = O[i];
          if (!(x.flags & FL_PRE) || !(x.flags & FL_REG)) continue;
          // register-partner table entries equal to the entry of their low bits
          // (after the op's 4 matrix entries and, with FL_THR, its 40 thread factors)
          const size_t f0 = x.data + 4 + ((x.flags & FL_THR) ? 40 : 0);
          const uint32_t lowmask = (1u << x.b0) - 1u;
          bool low = true;
          for (uint32_t idx = 0; idx < (1u << (RB - 1)) && low; ++idx) {
            const double2 u = D[f0 + idx], v = D[f0 + (idx & lowmask)];
            low = u.x == v.x && u.y == v.y;
          }
          if (low) x.flags |= FL_LOWF;
        }
        EncOp hp{};
        hp.type = OP_HPHASE;
        hp.b1 = (uint32_t)k;
        hp.flags = sc ? HPH_SCALE : 0u;
        hp.data = sc ? O[oe - 1].data : 0u;
        O.insert(O.begin() + (ptrdiff_t)ob, hp);
      }
    }
    sp.op_end = (uint32_t)O.size();
    sp.xload ^= carry_xload;
    carry_xload = 0;
    if (sp.op_end == sp.op_begin && &ph != &phases.back()) {
      // no op left (all folded): its flips move to the next phase's load
      carry_xload = sp.xload;
      continue;
    }
    last_tb = tb;
    last_regs = regs;
    P.push_back(sp);
  }
  if (SL.size() > (size_t)kMaxSlots) return fail(DQ_ERR_INTERNAL, "too many per-tile slots");

  for (const SwPhase& sp : P) {
    for (int i = 0; i < 32; ++i)
      if (sp.lanesw[i] >= (1u << m)) return fail(DQ_ERR_INTERNAL, "thread index outside the tile");
    for (int i = 0; i < 8; ++i)
      if (sp.warpsw[i] >= (1u << m)) return fail(DQ_ERR_INTERNAL, "thread index outside the tile");
    for (uint32_t b = 0; b < RB; ++b)
      if (sp.V[b] >= (1u << m)) return fail(DQ_ERR_INTERNAL, "register bit outside the tile");
  }
  for (const EncOp& so : O)
    if (((so.type <= OP_U2 || so.type == OP_U1H || so.type == OP_FLUSH_R) && so.b0 >= RB) ||
        (so.type == OP_FLUSH_T && so.b0 >= (uint32_t)kSwTB) || (so.type == OP_U2 && so.b1 >= RB) ||
        so.slot >= SL.size() + (SL.empty() ? 1 : 0) || so.data > std::max(D.size(), DS.size()) ||
        so.slot > 0xffffu ||
        so.creg > 0xffu || so.ctl_thr > 0xffu || so.flags > 0xffu)
      return fail(DQ_ERR_INTERNAL, "op encoding out of range");
  std::vector<SwOp> OP(O.size());
  for (size_t i = 0; i < O.size(); ++i) {
    const EncOp& e = O[i];
    OP[i].w0 = e.type | (e.b0 << 8) | (e.b1 << 16) | (e.creg << 24);
    OP[i].w1 = e.ctl_thr | (e.flags << 8) | (e.slot << 16);
    OP[i].data = e.data + (i < in_ds.size() && in_ds[i] ? (uint32_t)D.size() : 0u);
    OP[i].cnl = e.cnl;
  }
  SwHeader h{};
  h.m = m;
  h.rb = RB;
  // runs of 2^run_bits: the sweep's lowest run_bits local bits are qubits 0..run_bits-1
  uint32_t run_bits = 0;
  while (run_bits < 5 && run_bits < m && sw.local[run_bits] == run_bits) ++run_bits;
  run_bits = run_bits >= 5 ? 5u : 3u;
  if (m < run_bits || sw.local[run_bits - 1] != run_bits - 1)
    return fail(DQ_ERR_INTERNAL, "sweep local set lacks the pinned low qubits");
  h.run_bits = run_bits;
  const uint32_t nruns = 1u << (m - run_bits);
  std::vector<uint64_t> runoff(nruns);
  std::vector<uint32_t> runswz(nruns);
  for (uint32_t r = 0; r < nruns; ++r) {
    uint64_t off = 0;
    for (uint32_t b = 0; b + run_bits < m; ++b)
      if ((r >> b) & 1u) off |= 1ULL << sw.local[run_bits + b];
    runoff[r] = off;
    runswz[r] = swz(r << run_bits);
  }
  h.nphase = (uint32_t)P.size();
  h.nslots = (uint32_t)SL.size();
  {
    // every phase a straight-line phase: Hadamard-pattern sub-ops only, or
    // real 2x2 sub-ops only, select a restricted build
    bool marked = !P.empty(), had = false, real = false;
    for (const SwPhase& sp : P)
      if (sp.op_begin >= sp.op_end || O[sp.op_begin].type != OP_HPHASE) marked = false;
    for (const EncOp& e : O) {
      had = had || e.type == OP_U1H;
      real = real || e.type == OP_U1R;
    }
    const bool honly = marked && !real;
    h.flags = honly ? SWF_HONLY : (marked && !had ? SWF_RONLY : 0u);
    bool uonly = !P.empty() && !marked;
    for (const EncOp& e : O)
      if (!(e.type == OP_U1 || e.type == OP_U1R || e.type == OP_U1X) || (e.flags & FL_PRE)) uonly = false;
    if (uonly || !MP.empty()) h.flags = SWF_UONLY;
  }
  h.tile_xload = tile_xload;
  for (uint32_t k = 0; k < m; ++k) h.local_pos[k] = sw.local[k];
  const size_t hoff = blob.put(&h, 1);
  const size_t po = blob.put(P.data(), P.size());
  const size_t so = SL.empty() ? blob.align16() : blob.put(SL.data(), SL.size());
  const size_t eo = SE.empty() ? blob.align16() : blob.put(SE.data(), SE.size());
  const size_t ro = blob.put(runoff.data(), runoff.size());
  const size_t rs = blob.put(runswz.data(), runswz.size());
  // The last phase writes straight to the state when its lanes 0..2 are local
  // bits 0..2 (qubits 0..2): every 8-lane group then writes one 128-byte run.
  size_t go = 0;
  if (!P.empty() && last_tb.size() >= 3 && last_tb[0] == 0 && last_tb[1] == 1 && last_tb[2] == 2 &&
      sw.local[0] == 0 && sw.local[1] == 1 && sw.local[2] == 2) {
    SwGStore g{};
    for (uint32_t ln = 0; ln < 32; ++ln)
      for (int i = 0; i < 5; ++i)
        if ((ln >> i) & 1u) g.glane[ln] |= 1ULL << sw.local[last_tb[i]];
    for (uint32_t wp = 0; wp < 8; ++wp)
      for (int i = 0; i + 5 < kSwTB; ++i)
        if ((wp >> i) & 1u) g.gwarp[wp] |= 1ULL << sw.local[last_tb[5 + i]];
    for (uint32_t b = 0; b < RB && b < 4; ++b) g.gV[b] = 1ULL << sw.local[last_regs[b]];
    go = blob.put(&g, 1);
  }
  if (!MP.empty() && !go) return fail(DQ_ERR_INTERNAL, "the last rotation phase cannot write the state");
  // what the kernel of rotation phases does not need comes last: the general
  // ops and their data (DS continues D)
  const size_t mo = MP.empty() ? 0 : blob.put(MP.data(), MP.size());
  const size_t fo = FN.empty() ? blob.align16() : blob.put(FN.data(), FN.size());
  size_t oo = blob.align16();
  if (MP.empty() && !OP.empty()) oo = blob.put(OP.data(), OP.size());
  const size_t dd = D.empty() ? blob.align16() : blob.put(D.data(), D.size());
  const size_t stage = blob.align16() - hoff;
  if (!DS.empty()) blob.put(DS.data(), DS.size());
  if (!MP.empty() && !OP.empty()) oo = blob.put(OP.data(), OP.size());
  SwHeader* hp = reinterpret_cast<SwHeader*>(blob.buf.data() + hoff);
  hp->off_micro = mo ? (uint32_t)(mo - hoff) : 0u;
  hp->off_final = (uint32_t)(fo - hoff);
  hp->off_runoff = (uint32_t)(ro - hoff);
  hp->off_runswz = (uint32_t)(rs - hoff);
  hp->off_gstore = go ? (uint32_t)(go - hoff) : 0u;
  hp->off_phase = (uint32_t)(po - hoff);
  hp->off_op = (uint32_t)(oo - hoff);
  hp->off_slot = (uint32_t)(so - hoff);
  hp->off_slotent = (uint32_t)(eo - hoff);
  hp->off_data = (uint32_t)(dd - hoff);
  blob.align16();
  hp = reinterpret_cast<SwHeader*>(blob.buf.data() + hoff);
  hp->prog_bytes = (uint32_t)(blob.buf.size() - hoff);
  hp->stage_bytes = mo ? (uint32_t)stage : hp->prog_bytes;
  if (hp->stage_bytes > (uint32_t)max_prog((int)m)) return fail(DQ_ERR_INTERNAL, "sweep program too large");
  *offset = hoff;
  return DQ_OK;
}

// ---- gate conversion ----------------------------------------------------------------

// Convert one instruction (logical qubits mapped through perm) into planner
// gates.  Returns false if the fused path cannot represent it.
bool convert_inst(const dq_inst& in, const uint32_t* perm, std::vector<PGate>& out,
                  uint32_t* swap_a, uint32_t* swap_b, bool* is_swap) {
  *is_swap = false;
  hc u[4];
  auto diag1 = [&](uint32_t t, hc u00, hc u11, uint64_t ctrl) -> bool {
    // diag(u00, u11) on t with <= 1 control; returns false for more controls
    PGate g;
    g.kind = PG_DIAG;
    const int nc = __builtin_popcountll(ctrl);
    if (nc > 1 || !is_unit_phase(u00) || !is_unit_phase(u11)) return false;
    const hc rel = (u00.re == 1.0 && u00.im == 0.0) ? u11 : u11 * conj(u00);
    if (nc == 0) {
      if (!(u00.re == 1.0 && u00.im == 0.0)) g.cst = u00;
      g.nlin = 1;
      g.lq[0] = t;
      g.lw[0] = rel;
      g.touched = 1ULL << t;
    } else {
      const uint32_t c = (uint32_t)__builtin_ctzll(ctrl);
      if (!(u00.re == 1.0 && u00.im == 0.0)) {
        g.nlin = 1;
        g.lq[0] = c;
        g.lw[0] = u00;
      }
      g.quad = true;
      g.qa = c;
      g.qb = t;
      g.qw = rel;
      g.touched = (1ULL << t) | ctrl;
    }
    out.push_back(g);
    return true;
  };
  auto u1 = [&](uint32_t t, const hc* m, uint64_t ctrl, bool xperm) {
    PGate g;
    g.kind = xperm ? PG_U1X : PG_U1;
    g.t0 = t;
    g.ctrl = ctrl;
    for (int i = 0; i < 4; ++i) g.u[i] = m[i];
    g.real = !xperm && m[0].im == 0.0 && m[1].im == 0.0 && m[2].im == 0.0 && m[3].im == 0.0;
    g.had = g.real && ctrl == 0 && m[0].re == m[1].re && m[0].re == m[2].re &&
            m[0].re == -m[3].re;
    g.touched = (1ULL << t) | ctrl;
    out.push_back(g);
  };
  if (matrix_1q(in.kind, in.p, u)) {
    const uint32_t t = perm[in.q[0]];
    if (is_zero(u[1]) && is_zero(u[2]) && diag1(t, u[0], u[3], 0)) return true;
    const bool xp = is_zero(u[0]) && is_zero(u[3]) && is_one(u[1]) && is_one(u[2]);
    u1(t, u, 0, xp);
    return true;
  }
  Gate g;
  if (!matrix_nq(in, g)) return false;
  for (uint32_t b = 0; b < g.k; ++b) g.qubits[b] = perm[g.qubits[b]];
  GateOp op;
  classify(g, op);
  switch (op.cls) {
    case GC_PHASE: {
      const hc one{1, 0};
      if (__builtin_popcountll(op.ctrl_mask) <= 1 && diag1(op.target, one, op.u[0], op.ctrl_mask))
        return true;
      hc m[4] = {one, hc{0, 0}, hc{0, 0}, op.u[0]};
      u1(op.target, m, op.ctrl_mask, false);
      return true;
    }
    case GC_ONE_Q:
      if (is_zero(op.u[1]) && is_zero(op.u[2]) && __builtin_popcountll(op.ctrl_mask) <= 1 &&
          diag1(op.target, op.u[0], op.u[3], op.ctrl_mask))
        return true;
      u1(op.target, op.u, op.ctrl_mask, false);
      return true;
    case GC_XPERM: {
      hc m[4] = {hc{0, 0}, hc{1, 0}, hc{1, 0}, hc{0, 0}};
      u1(op.target, m, op.ctrl_mask, true);
      return true;
    }
    case GC_SWAP: {
      if (op.ctrl_mask == 0) {
        *is_swap = true;
        // logical qubits of the swap (relabel the logical -> physical map)
        *swap_a = (uint32_t)in.q[in.nq - 2];
        *swap_b = (uint32_t)in.q[in.nq - 1];
        return true;
      }
      // controlled swap = cx(b->a) . ccx(c, a -> b) . cx(b->a), exact permutations
      const uint32_t a = op.target, b = op.target2;
      hc xm[4] = {hc{0, 0}, hc{1, 0}, hc{1, 0}, hc{0, 0}};
      u1(a, xm, (1ULL << b), true);
      u1(b, xm, op.ctrl_mask | (1ULL << a), true);
      u1(a, xm, (1ULL << b), true);
      return true;
    }
    case GC_DIAG: {
      if (g.k != 2) return false;
      const hc d00 = g.m[0], d01 = g.m[5], d10 = g.m[10], d11 = g.m[15];
      if (!is_unit_phase(d00) || !is_unit_phase(d01) || !is_unit_phase(d10) || !is_unit_phase(d11))
        return false;
      PGate p;
      p.kind = PG_DIAG;
      const uint32_t qa = g.qubits[0], qb = g.qubits[1];
      p.cst = d00;
      p.nlin = 2;
      p.lq[0] = qa;
      p.lw[0] = d10 * conj(d00);
      p.lq[1] = qb;
      p.lw[1] = d01 * conj(d00);
      p.quad = true;
      p.qa = qa;
      p.qb = qb;
      p.qw = d11 * d00 * conj(d01) * conj(d10);
      p.touched = (1ULL << qa) | (1ULL << qb);
      out.push_back(p);
      return true;
    }
    case GC_DENSE: {
      if (g.k != 2) return false;
      PGate p;
      p.kind = PG_U2;
      p.t0 = g.qubits[0];
      p.t1 = g.qubits[1];
      for (int i = 0; i < 16; ++i) p.u[i] = g.m[i];
      p.touched = (1ULL << p.t0) | (1ULL << p.t1);
      out.push_back(p);
      return true;
    }
    default:
      return false;
  }
}

template <int TB, int RB, int S, int RUNB, int FORM = FORM_ALL>
int launch_sweep_r(double2* amp, uint32_t n, const uint8_t* dblob, uint32_t prog_bytes,
                   cudaStream_t st, long long synth) {
  constexpr int M = TB + RB;
  const size_t smem_max = sizeof(double2) * (S * (1u << M) + kMaxSlots) + max_prog(M);
  const size_t smem = sizeof(double2) * (S * (1u << M) + kMaxSlots) + prog_bytes;
  // per device, once: opt-in shared memory; resident CTAs per SM for this
  // launch's shared memory (programs are mostly far below the maximum), cached
  // per 4 KB of program size (the mutex makes concurrent host threads safe)
  static std::mutex mu;
  static bool attr_done[64];
  static int per_sm[64][17];  // 0 = not yet queried
  int dev = 0;
  DQ_CUDA_TRY(cudaGetDevice(&dev));
  int resident;
  {
    std::lock_guard<std::mutex> lk(mu);
    if (!attr_done[dev & 63]) {
      DQ_CUDA_TRY(cudaFuncSetAttribute(k_sweep<TB, RB, S, RUNB, FORM>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_max));
      attr_done[dev & 63] = true;
    }
    const uint32_t bucket = std::min<uint32_t>(16, (prog_bytes + 4095) / 4096);
    const size_t smem_b = std::min(smem_max, smem - prog_bytes + 4096 * (size_t)bucket);
    int& r = per_sm[dev & 63][bucket];
    if (r == 0) {
      int b = 1;
      DQ_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_sweep<TB, RB, S, RUNB, FORM>,
                                                                1 << TB, smem_b));
      r = b < 1 ? 1 : b;
    }
    resident = r;
  }
  int sms = 148;
  DQ_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const uint64_t tiles = 1ULL << (n - M);
  const unsigned grid = (unsigned)std::min<uint64_t>(tiles, (uint64_t)sms * resident);
  k_sweep<TB, RB, S, RUNB, FORM><<<grid, 1 << TB, smem, st>>>(amp, dblob, prog_bytes, (uint32_t)tiles,
                                                               synth);
  DQ_CUDA_TRY(cudaGetLastError());
  return DQ_OK;
}

// DQSIM_SWEEP_STAGES=2: double-buffered tiles
int sweep_stages() {
  static const int stages = [] {
    const char* e = getenv("DQSIM_SWEEP_STAGES");
    return e ? atoi(e) : 1;
  }();
  return stages;
}

template <int TB, int RB>
int launch_sweep_rb(double2* amp, uint32_t n, const uint8_t* dblob, uint32_t prog_bytes,
                    cudaStream_t st, long long synth, uint32_t run_bits, uint32_t flags, bool micro) {
  // default: single-buffered tiles, three 128-thread CTAs per SM (measured
  // faster than two double-buffered CTAs: the extra warps hide more of the
  // per-op latency than the prefetch saves); DQSIM_SWEEP_STAGES=2 selects
  // double buffering
  if (TB == 7 && sweep_stages() != 2) {
    if (RB == 4 && micro)
      return run_bits == 3 ? launch_sweep_r<7, 4, 1, 3, FORM_M>(amp, n, dblob, prog_bytes, st, synth)
                           : launch_sweep_r<7, 4, 1, 5, FORM_M>(amp, n, dblob, prog_bytes, st, synth);
    if (RB == 4 && (flags & SWF_HONLY))
      return run_bits == 3 ? launch_sweep_r<7, 4, 1, 3, FORM_H>(amp, n, dblob, prog_bytes, st, synth)
                           : launch_sweep_r<7, 4, 1, 5, FORM_H>(amp, n, dblob, prog_bytes, st, synth);
    if (RB == 4 && (flags & SWF_RONLY))
      return run_bits == 3 ? launch_sweep_r<7, 4, 1, 3, FORM_R>(amp, n, dblob, prog_bytes, st, synth)
                           : launch_sweep_r<7, 4, 1, 5, FORM_R>(amp, n, dblob, prog_bytes, st, synth);
    if (RB == 4 && (flags & SWF_UONLY))
      return run_bits == 3 ? launch_sweep_r<7, 4, 1, 3, FORM_U>(amp, n, dblob, prog_bytes, st, synth)
                           : launch_sweep_r<7, 4, 1, 5, FORM_U>(amp, n, dblob, prog_bytes, st, synth);
    return run_bits == 3 ? launch_sweep_r<7, RB, 1, 3>(amp, n, dblob, prog_bytes, st, synth)
                         : launch_sweep_r<7, RB, 1, 5>(amp, n, dblob, prog_bytes, st, synth);
  }
  return run_bits == 3 ? launch_sweep_r<TB, RB, 2, 3>(amp, n, dblob, prog_bytes, st, synth)
                       : launch_sweep_r<TB, RB, 2, 5>(amp, n, dblob, prog_bytes, st, synth);
}

int launch_sweep(double2* amp, uint32_t n, uint32_t TB, uint32_t RB, const uint8_t* dblob,
                 uint32_t prog_bytes, cudaStream_t st, long long synth, uint32_t run_bits,
                 uint32_t flags, bool micro) {
  if (TB == 8) {
    switch (RB) {
      case 2: return launch_sweep_rb<8, 2>(amp, n, dblob, prog_bytes, st, synth, run_bits, flags, micro);
      case 3: return launch_sweep_rb<8, 3>(amp, n, dblob, prog_bytes, st, synth, run_bits, flags, micro);
      case 4: return launch_sweep_rb<8, 4>(amp, n, dblob, prog_bytes, st, synth, run_bits, flags, micro);
      default: break;
    }
  } else if (TB == 7) {
    switch (RB) {
      case 2: return launch_sweep_rb<7, 2>(amp, n, dblob, prog_bytes, st, synth, run_bits, flags, micro);
      case 3: return launch_sweep_rb<7, 3>(amp, n, dblob, prog_bytes, st, synth, run_bits, flags, micro);
      case 4: return launch_sweep_rb<7, 4>(amp, n, dblob, prog_bytes, st, synth, run_bits, flags, micro);
      default: break;
    }
  }
  return fail(DQ_ERR_INTERNAL, "unsupported sweep geometry");
}

template <int TB, int RB, int RUNB, int FORM = FORM_ALL>
int launch_sweep_multi_t(const SweepJob* d_jobs, uint32_t njobs, uint32_t n, uint32_t max_bytes,
                         cudaStream_t st) {
  constexpr int M = TB + RB;
  const size_t smem_max = sizeof(double2) * ((1u << M) + kMaxSlots) + max_prog(M);
  const size_t smem = sizeof(double2) * ((1u << M) + kMaxSlots) + max_bytes;
  // resident CTAs per SM for this launch's shared memory, cached per 4 KB of
  // program size (programs are mostly far below the maximum)
  static std::mutex mu;
  static bool attr_done[64];
  static int per_sm[64][17];
  int dev = 0;
  DQ_CUDA_TRY(cudaGetDevice(&dev));
  int resident;
  {
    std::lock_guard<std::mutex> lk(mu);
    if (!attr_done[dev & 63]) {
      DQ_CUDA_TRY(cudaFuncSetAttribute(k_sweep_multi<TB, RB, RUNB, FORM>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_max));
      attr_done[dev & 63] = true;
    }
    const uint32_t bucket = std::min<uint32_t>(16, (max_bytes + 4095) / 4096);
    const size_t smem_b = std::min(smem_max, smem - max_bytes + 4096 * (size_t)bucket);
    int& r = per_sm[dev & 63][bucket];
    if (r == 0) {
      int b = 1;
      DQ_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_sweep_multi<TB, RB, RUNB, FORM>,
                                                                1 << TB, smem_b));
      r = b < 1 ? 1 : b;
    }
    resident = r;
  }
  int sms = 148;
  DQ_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const uint32_t ntiles = 1u << (n - M);
  const uint32_t chunk = std::min<uint32_t>(64, ntiles);
  const uint32_t nchunks = (ntiles + chunk - 1) / chunk;
  const uint64_t work = (uint64_t)njobs * nchunks;
  const unsigned grid = (unsigned)std::min<uint64_t>(work, (uint64_t)sms * resident);
  k_sweep_multi<TB, RB, RUNB, FORM><<<grid, 1 << TB, smem, st>>>(d_jobs, njobs, nchunks, chunk, ntiles);
  DQ_CUDA_TRY(cudaGetLastError());
  return DQ_OK;
}

int ensure_capacity(FusedWork& fw, size_t bytes, cudaStream_t st) {
  if (bytes <= fw.d_cap && bytes <= fw.h_cap) return DQ_OK;
  DQ_CUDA_TRY(cudaStreamSynchronize(st));
  size_t cap = std::max<size_t>(bytes, 1 << 16);
  cap = std::max(cap, fw.d_cap * 2);
  if (fw.d_blob) cudaFree(fw.d_blob);
  if (fw.h_blob) cudaFreeHost(fw.h_blob);
  fw.d_blob = nullptr;
  fw.h_blob = nullptr;
  fw.d_cap = fw.h_cap = 0;
  DQ_CUDA_TRY(cudaMalloc((void**)&fw.d_blob, cap));
  DQ_CUDA_TRY(cudaMallocHost((void**)&fw.h_blob, cap));
  fw.d_cap = fw.h_cap = cap;
  return DQ_OK;
}

}  // namespace

void fused_release(FusedWork& fw) {
  if (fw.d_blob) cudaFree(fw.d_blob);
  if (fw.h_blob) cudaFreeHost(fw.h_blob);
  for (auto e : fw.events) cudaEventDestroy(e);
  fw = FusedWork();
}

// ---- relabel materialisation ------------------------------------------------------------

int materialize_perm(double2* amp, uint32_t n, uint32_t* perm, cudaStream_t st, uint64_t* launches) {
  // sigma(p) = logical qubit stored at physical p: data bit p moves to sigma(p)
  uint32_t sigma[64];
  bool ident = true;
  for (uint32_t l = 0; l < n; ++l) {
    sigma[perm[l]] = l;
    if (perm[l] != l) ident = false;
  }
  if (ident) return DQ_OK;
  // sigma = tau2 o tau1, both involutions (cycle reflections)
  uint32_t tau1[64], tau2[64];
  for (uint32_t p = 0; p < n; ++p) tau1[p] = tau2[p] = p;
  std::vector<char> seen(n, 0);
  for (uint32_t p = 0; p < n; ++p) {
    if (seen[p]) continue;
    std::vector<uint32_t> cyc;
    uint32_t x = p;
    while (!seen[x]) {
      seen[x] = 1;
      cyc.push_back(x);
      x = sigma[x];
    }
    const size_t k = cyc.size();
    for (size_t i = 0; i < k; ++i) {
      tau1[cyc[i]] = cyc[(k - i) % k];
      tau2[cyc[i]] = cyc[(k + 1 - i) % k];
    }
  }
  const uint32_t* taus[2] = {tau1, tau2};
  for (int r = 0; r < 2; ++r) {
    const uint32_t* tau = taus[r];
    bool id = true;
    for (uint32_t p = 0; p < n; ++p)
      if (tau[p] != p) id = false;
    if (id) continue;
    // local set: closed under tau, the lowest positions with their images
    uint64_t L = 0;
    for (uint32_t p = 0; p < n; ++p) {
      const uint64_t add = (1ULL << p) | (1ULL << tau[p]);
      if ((uint32_t)__builtin_popcountll(L | add) <= kPermBits) L |= add;
    }
    PermParams P{};
    P.n = n;
    uint32_t pos[kPermBits];  // element bit -> position
    int li[64];
    for (uint32_t p = 0; p < 64; ++p) {
      P.tau[p] = (uint8_t)(p < n ? tau[p] : p);
      P.from[p] = 63;
      li[p] = -1;
      if (p < n && (L >> p & 1ULL)) {
        li[p] = (int)P.m;
        pos[P.m++] = p;
      }
    }
    // consecutive tiles differ in the lowest remaining positions and their
    // images, so that neighbouring warps touch neighbouring memory on both sides
    uint8_t next = 0;
    for (uint32_t p = 0; p < n; ++p) {
      if ((L >> p & 1ULL) || P.from[p] != 63) continue;
      P.from[p] = next++;
      if (tau[p] != p) P.from[tau[p]] = next++;
    }
    for (uint32_t b = 0; b < P.m; ++b) {
      const uint32_t img = 1u << li[tau[pos[b]]];
      if (b < 5) {
        P.lane_d[b] = 1ULL << pos[b];
        P.lane_t[b] = img;
      } else {
        for (uint32_t i = 0; i < 8; ++i)
          if (i >> (b - 5) & 1u) {
            P.di[i] |= 1ULL << pos[b];
            P.ti[i] |= img;
          }
      }
    }
    constexpr size_t smem = sizeof(double2) * kPermWarps * 2 * (1u << kPermBits);
    static std::mutex mu;
    static uint64_t attr_done = 0;  // one bit per device
    int dev = 0, sms = 148;
    DQ_CUDA_TRY(cudaGetDevice(&dev));
    DQ_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    {
      std::lock_guard<std::mutex> lk(mu);
      if (!((attr_done >> (dev & 63)) & 1ULL)) {
        DQ_CUDA_TRY(cudaFuncSetAttribute(k_permute_pairs, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem));
        attr_done |= 1ULL << (dev & 63);
      }
    }
    const uint64_t tiles = 1ULL << (n - P.m);
    const unsigned grid = (unsigned)std::min<uint64_t>((tiles + kPermWarps - 1) / kPermWarps, 3ULL * sms);
    k_permute_pairs<<<grid, 32 * kPermWarps, smem, st>>>(amp, P, tiles);
    DQ_CUDA_TRY(cudaGetLastError());
    if (launches) ++*launches;
  }
  for (uint32_t l = 0; l < n; ++l) perm[l] = l;
  return DQ_OK;
}

// ---- program runner ------------------------------------------------------------------------

int fused_run_segment(double2* amp, uint32_t n, std::vector<PGate>& G, Planner& pl, Poly& poly,
                      FusedWork& fw, cudaStream_t st, bool timing, dq_profile* prof,
                      int64_t* lazy_basis) {
  std::vector<PSweep> sweeps;
  Blob blob;
  std::vector<size_t> offs;
  auto encode = [&]() -> int {
    blob.buf.clear();
    offs.assign(sweeps.size(), 0);
    for (size_t i = 0; i < sweeps.size(); ++i)
      DQ_TRY(encode_sweep(sweeps[i], G, pl.TB, pl.RB, blob, &offs[i], fw.plan_out && !fw.plan_tb));
    return DQ_OK;
  };
  // one pass of the planner with the given low qubits pinned
  bool micro = pl.micro_ok && poly.empty() && !poly.has_cst && micro_eligible(G);
  auto plan_with = [&](uint64_t pinned, Poly& p, std::vector<PSweep>& out) {
    pl.pinned = pinned;
    out.clear();
    pl.plan(G, p, out);
    pl.final_flush(p, out);
  };
  const uint64_t pin0 = pl.pinned;
  if (micro) {
    // rotation phases are cheap enough that the two more tile qubits of
    // 128-byte runs always save sweeps (28-qubit brickwork: 30 against 45)
    if (pl.pin_auto) pl.pinned = 0x7ULL;
    MicroPlanner mp{pl};
    mp.split(G);
    PolyX px;  // a segment starts without pending terms
    px.init(pl.n);
    if (mp.ok) mp.plan(px, sweeps);
    micro = !sweeps.empty();  // no plan: not all gates are unitary, or none needs a sweep
    if (micro) {
      mp.final_flush(px, sweeps);
      if (encode() != DQ_OK) {  // planned as general ops instead
        clear_error();
        micro = false;
      }
    }
    pl.pinned = pin0;
  }
  if (!micro) {
    if (pl.pin_auto && !pl.single_tile) {
      // plan with qubits 0..4 pinned and with 0..2 pinned; the wider tile
      // choice wins only when it saves at least a tenth of the sweeps (its
      // 128-byte runs cost a little more per sweep)
      Poly poly3 = poly;
      std::vector<PSweep> sweeps3;
      plan_with(0x1FULL, poly, sweeps);
      plan_with(0x7ULL, poly3, sweeps3);
      if (10 * sweeps3.size() <= 9 * sweeps.size()) {
        sweeps.swap(sweeps3);
        poly = poly3;
      }
    } else {
      plan_with(pin0, poly, sweeps);
    }
    if (sweeps.empty()) return DQ_OK;
    DQ_TRY(encode());
  }
  blob.align16();
  if (fw.plan_out) {  // plan-only: hand the programs back instead of running them
    const size_t base = fw.plan_out->size();
    fw.plan_out->insert(fw.plan_out->end(), blob.buf.begin(), blob.buf.end());
    for (size_t o : offs) fw.plan_offs->push_back(base + o);
    fw.plan_rb = pl.RB;
    if (lazy_basis && *lazy_basis >= 0) {  // the first sweep generates the basis vector
      fw.plan_synth = *lazy_basis;
      *lazy_basis = -1;
    }
    prof->sweeps += sweeps.size();
    return DQ_OK;
  }
  // the pinned staging buffer may still feed an earlier copy
  DQ_CUDA_TRY(cudaStreamSynchronize(st));
  DQ_TRY(ensure_capacity(fw, blob.buf.size(), st));
  memcpy(fw.h_blob, blob.buf.data(), blob.buf.size());
  DQ_CUDA_TRY(cudaMemcpyAsync(fw.d_blob, fw.h_blob, blob.buf.size(), cudaMemcpyHostToDevice, st));
  for (size_t i = 0; i < sweeps.size(); ++i) {
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (timing) {
      cudaEventCreate(&e0);
      cudaEventCreate(&e1);
      cudaEventRecord(e0, st);
    }
    const SwHeader* hh = reinterpret_cast<const SwHeader*>(blob.buf.data() + offs[i]);
    // a pending basis state is consumed by the first sweep (it writes every amplitude)
    const long long synth = (lazy_basis && *lazy_basis >= 0) ? (long long)*lazy_basis : -1;
    DQ_TRY(launch_sweep(amp, n, pl.TB, pl.RB, fw.d_blob + offs[i], hh->stage_bytes, st, synth,
                        hh->run_bits, hh->flags, hh->off_micro != 0));
    if (lazy_basis) *lazy_basis = -1;
    if (timing) {
      cudaEventRecord(e1, st);
      fw.events.push_back(e0);
      fw.events.push_back(e1);
    }
    ++prof->sweeps;
    ++prof->kernel_launches;
  }
  return DQ_OK;
}

int fused_run(double2* amp, uint32_t n, const dq_inst* prog, uint64_t ninst, const dq_run_opts& o,
              FusedWork& fw, cudaStream_t st, int device, FusedHooks& hooks, dq_profile* prof,
              uint32_t* perm) {
  (void)device;
  Planner pl;
  pl.n = n;
  // thread geometry: DQSIM_SWEEP_TB=8 selects one 256-thread CTA per SM
  static const uint32_t tb_env = []() {
    const char* e = getenv("DQSIM_SWEEP_TB");
    return (e && atoi(e) == 8) ? 8u : 7u;
  }();
  const uint32_t TB = fw.plan_tb ? fw.plan_tb : tb_env;
  uint32_t M = TB + 4;  // 16 amplitudes per thread
  if (o.fusion_width >= (int)(TB + 2) && o.fusion_width <= (int)(TB + 4)) M = (uint32_t)o.fusion_width;
  if (M > n) M = n;
  pl.M = M;
  pl.TB = TB;
  pl.RB = M - TB;
  pl.single_tile = (M == n);
  // the trajectory launch runs 8-thread-bit plans, k_sweep and k_sweep_multi 7-bit ones
  pl.micro_ok = pl.RB == 4 && (TB == 7 ? sweep_stages() != 2 : fw.plan_tb != 0);
  // Pinned tile qubits: 0..4 (512-byte runs) or 0..2 (128-byte runs, two
  // more tile qubits free); by default each segment of 20+ qubits is planned
  // both ways and keeps the one with clearly fewer sweeps.
  // DQSIM_SWEEP_PIN=5 / 3 forces one.
  static const int pin_env = []() {
    const char* e = getenv("DQSIM_SWEEP_PIN");
    return e ? atoi(e) : 0;
  }();
  pl.pinned = pin_env == 3 ? 0x7ULL : 0x1FULL;
  pl.pin_auto = pin_env == 0 && n >= 20;
  if (o.max_cost > 0) pl.budget = (double)o.max_cost;
  Poly poly;
  poly.init(n);
  for (auto e : fw.events) cudaEventDestroy(e);
  fw.events.clear();
  const bool timing = o.time_sweeps != 0;

  // shots semantics: run the reference's fuse_circuit output
  std::vector<FusedEntry> fe;
  if (o.semantics == DQ_SEM_SHOTS) {
    fe = fuse_program(prog, ninst, n);
  } else {
    fe.resize(ninst);
    for (uint64_t i = 0; i < ninst; ++i) fe[i].inst = (int64_t)i;
  }

  std::vector<PGate> G;
  auto flush_segment = [&]() -> int {
    if (G.empty() && poly.empty()) return DQ_OK;
    int rc = fused_run_segment(amp, n, G, pl, poly, fw, st, timing, prof, hooks.lazy_basis);
    G.clear();
    return rc;
  };
  for (const FusedEntry& e : fe) {
    if (e.inst < 0) {  // a fused 2x2 of the shots path
      PGate g;
      const uint32_t t = perm[e.qubit];
      if (is_zero(e.m[1]) && is_zero(e.m[2]) && is_unit_phase(e.m[0]) && is_unit_phase(e.m[3])) {
        g.kind = PG_DIAG;
        if (!(e.m[0].re == 1.0 && e.m[0].im == 0.0)) g.cst = e.m[0];
        g.nlin = 1;
        g.lq[0] = t;
        g.lw[0] = (e.m[0].re == 1.0 && e.m[0].im == 0.0) ? e.m[3] : e.m[3] * conj(e.m[0]);
      } else {
        g.kind = PG_U1;
        g.t0 = t;
        for (int k = 0; k < 4; ++k) g.u[k] = e.m[k];
        g.real = e.m[0].im == 0.0 && e.m[1].im == 0.0 && e.m[2].im == 0.0 && e.m[3].im == 0.0;
      }
      g.touched = 1ULL << t;
      G.push_back(g);
      continue;
    }
    const dq_inst& in = prog[e.inst];
    const int64_t src = e.inst;
    // conditions are final: no measurement inside a segment
    bool ok = true;
    for (uint32_t c = 0; c < in.cond_count && ok; ++c) {
      const dq_cond& cd = hooks.conds[in.cond_first + c];
      uint64_t actual = 0;
      for (uint64_t b = 0; b < cd.creg_size; ++b) {
        const uint64_t idx = cd.creg_base + b;
        const uint64_t v = (idx < hooks.ncbits && hooks.cbits[idx] > 0) ? (uint64_t)hooks.cbits[idx] : 0;
        actual |= v << b;
      }
      ok = (actual == cd.creg_value);
    }
    if (!ok) continue;
    // While the state is still a pending basis vector and nothing has been
    // queued yet, an X gate is a flip of that basis index: exact, and it
    // leaves every tile qubit free for the gates that follow.
    if (in.kind == DQ_X && hooks.lazy_basis && *hooks.lazy_basis >= 0 && G.empty() &&
        poly.empty() && !poly.has_cst) {
      *hooks.lazy_basis ^= (int64_t)(1ULL << perm[in.q[0]]);
      continue;
    }
    switch (in.kind) {
      case DQ_ID: case DQ_U0: case DQ_BARRIER: case DQ_CLASSICAL: case DQ_G_NOOP:
        continue;
      case DQ_G_OPAQUE:
        if (o.semantics == DQ_SEM_SHOTS) continue;
        prof->failed_inst = src;
        return fail(DQ_ERR_UNSUPPORTED, "unsupported generic gate");
      case DQ_G_UNSUPPORTED:
        prof->failed_inst = src;
        return fail(DQ_ERR_UNSUPPORTED, "unsupported generic gate");
      case DQ_MEASURE:
      case DQ_RESET: {
        if (fw.plan_out) return fail(DQ_ERR_INVALID_ARG, "plan-only mode takes unitary programs");
        DQ_TRY(flush_segment());
        int out = 0;
        DQ_TRY(hooks.measure(perm[in.q[0]], &out));
        if (in.kind == DQ_MEASURE) {
          hooks.cbits[in.cbit] = out;
        } else if (out == 1) {
          GateOp op;
          hc xm[4] = {hc{0, 0}, hc{1, 0}, hc{1, 0}, hc{0, 0}};
          classify_1q(xm, perm[in.q[0]], 0, op);
          DQ_TRY(hooks.exact_gate(op));
        }
        continue;
      }
      default:
        break;
    }
    uint32_t sa = 0, sb = 0;
    bool is_swap = false;
    const size_t before = G.size();
    if (convert_inst(in, perm, G, &sa, &sb, &is_swap)) {
      if (is_swap) std::swap(perm[sa], perm[sb]);
      continue;
    }
    G.resize(before);
    if (fw.plan_out) return fail(DQ_ERR_INVALID_ARG, "plan-only mode: gate not representable");
    // not representable in a sweep: flush, then the exact per-gate kernel
    DQ_TRY(flush_segment());
    GateOp op;
    hc u[4];
    if (matrix_1q(in.kind, in.p, u)) {
      classify_1q(u, perm[in.q[0]], 0, op);
    } else {
      Gate g;
      if (!matrix_nq(in, g)) return fail(DQ_ERR_INTERNAL, "instruction kind without a matrix");
      for (uint32_t b = 0; b < g.k; ++b) g.qubits[b] = perm[g.qubits[b]];
      classify(g, op);
    }
    DQ_TRY(hooks.exact_gate(op));
  }
  DQ_TRY(flush_segment());
  if (timing && !fw.plan_out) {
    DQ_CUDA_TRY(cudaStreamSynchronize(st));
    double t = 0;
    for (size_t i = 0; i + 1 < fw.events.size(); i += 2) {
      float ms = 0.f;
      cudaEventElapsedTime(&ms, fw.events[i], fw.events[i + 1]);
      t += ms * 1e-3;
    }
    prof->sweep_time += t;
  }
  return DQ_OK;
}

int fused_plan(uint32_t n, const dq_inst* prog, uint64_t ninst, int semantics, uint32_t tb,
               int fusion_width, int64_t lazy_basis, std::vector<uint8_t>* blob,
               std::vector<uint64_t>* offs, uint32_t* perm, int64_t* synth, uint32_t* rb) {
  if (n < kFusedMinQubits || n > 34) return fail(DQ_ERR_INVALID_ARG, "fused planning needs 10..34 qubits");
  FusedWork fw;
  fw.plan_out = blob;
  fw.plan_offs = offs;
  fw.plan_tb = tb;
  FusedHooks hooks;
  int64_t lazy = lazy_basis;
  hooks.lazy_basis = lazy_basis >= 0 ? &lazy : nullptr;
  dq_profile prof{};
  prof.failed_inst = -1;
  dq_run_opts o{};
  o.semantics = semantics;
  o.exec = DQ_EXEC_FUSED;
  o.fusion_width = fusion_width;
  DQ_TRY(fused_run(nullptr, n, prog, ninst, o, fw, nullptr, 0, hooks, &prof, perm));
  *synth = offs->empty() ? (lazy_basis >= 0 ? lazy : -1) : fw.plan_synth;
  *rb = fw.plan_rb;
  return DQ_OK;
}

uint32_t sweep_run_bits(const uint8_t* prog) {
  return reinterpret_cast<const SwHeader*>(prog)->run_bits;
}

uint32_t sweep_prog_bytes(const uint8_t* prog) {
  return reinterpret_cast<const SwHeader*>(prog)->stage_bytes;
}

uint32_t sweep_flags(const uint8_t* prog) {
  const SwHeader* h = reinterpret_cast<const SwHeader*>(prog);
  return h->off_micro ? SWF_MICRO : h->flags | SWF_OPS;
}

int launch_sweep_multi(const SweepJob* d_jobs, uint32_t njobs, uint32_t n, uint32_t rb,
                       uint32_t run_bits, uint32_t max_bytes, cudaStream_t st, uint32_t flags) {
  if (!njobs) return DQ_OK;
  if (n < 7 + rb) return fail(DQ_ERR_INVALID_ARG, "state smaller than a tile");
  if (max_bytes > (uint32_t)max_prog(7 + (int)rb)) return fail(DQ_ERR_INTERNAL, "sweep program too large");
  if (!(flags & (SWF_MICRO | SWF_OPS))) return fail(DQ_ERR_INTERNAL, "rotation phases and ops in one launch");
  const bool r3 = run_bits == 3;
  switch (rb) {
    case 2: return r3 ? launch_sweep_multi_t<7, 2, 3>(d_jobs, njobs, n, max_bytes, st)
                      : launch_sweep_multi_t<7, 2, 5>(d_jobs, njobs, n, max_bytes, st);
    case 3: return r3 ? launch_sweep_multi_t<7, 3, 3>(d_jobs, njobs, n, max_bytes, st)
                      : launch_sweep_multi_t<7, 3, 5>(d_jobs, njobs, n, max_bytes, st);
    case 4:
      // every job's program allows a restricted build (the flags of all of them ANDed)
      if (flags & SWF_MICRO)
        return r3 ? launch_sweep_multi_t<7, 4, 3, FORM_M>(d_jobs, njobs, n, max_bytes, st)
                  : launch_sweep_multi_t<7, 4, 5, FORM_M>(d_jobs, njobs, n, max_bytes, st);
      if (flags & SWF_HONLY)
        return r3 ? launch_sweep_multi_t<7, 4, 3, FORM_H>(d_jobs, njobs, n, max_bytes, st)
                  : launch_sweep_multi_t<7, 4, 5, FORM_H>(d_jobs, njobs, n, max_bytes, st);
      if (flags & SWF_RONLY)
        return r3 ? launch_sweep_multi_t<7, 4, 3, FORM_R>(d_jobs, njobs, n, max_bytes, st)
                  : launch_sweep_multi_t<7, 4, 5, FORM_R>(d_jobs, njobs, n, max_bytes, st);
      if (flags & SWF_UONLY)
        return r3 ? launch_sweep_multi_t<7, 4, 3, FORM_U>(d_jobs, njobs, n, max_bytes, st)
                  : launch_sweep_multi_t<7, 4, 5, FORM_U>(d_jobs, njobs, n, max_bytes, st);
      return r3 ? launch_sweep_multi_t<7, 4, 3>(d_jobs, njobs, n, max_bytes, st)
                : launch_sweep_multi_t<7, 4, 5>(d_jobs, njobs, n, max_bytes, st);
    default: return fail(DQ_ERR_INTERNAL, "unsupported multi-sweep geometry");
  }
}

}  // namespace dq
