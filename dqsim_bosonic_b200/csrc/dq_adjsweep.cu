// dq_adjsweep.cu — the adjoint backward pass as fused tile sweeps.
//
// The per-gate backward (dq_adjoint.cu) streams psi and lambda through HBM
// once per gate (64 B per amplitude per gate).  Here a sweep loads a tile of
// 2^m amplitudes of both vectors into shared memory (the tile spans the m
// "local" qubits: bits 0..2 for coalescing plus up to m - 3 chosen ones),
// applies a run of gates in reverse program order to both, reduces every
// gate's gradient terms, and writes the tile back: 64 B per amplitude per
// sweep instead of per gate.  A gate can join the current sweep when
//   * it is diagonal (any qubits: a non-local bit is constant over a tile), or
//   * its non-diagonal qubits (a one-qubit target, both qubits of a dense
//     two-qubit gate) are local — the planner widens the local set up to m.
// Gates of three or more qubits end the sweep and are undone by the exact
// per-gate kernels on both vectors (they carry no trainable parameter).
//
// Ops (all act on psi and lambda; V = U^dagger, D_j = dU/dtheta_j):
//   A_ONE   2x2 on a local target; optional local control mask; optional
//           non-local selector bit choosing between two matrix variants
//           (controlled gates with a non-local control: variant 0 = I).
//   A_TWO   dense 4x4 on two local qubits (rxx, swap-like, psi+-, phi+).
//   A_DIAG  diagonal on up to two qubits, local or not, applied elementwise.
//   A_PASS  header of a register pass: a thread holds the 8 amplitudes of psi
//           and lambda that differ in three local bits, applies a run of
//           diagonal gates on any qubits (diag_grads, diag_apply), then up to
//           three rotations of one form on those bits (pass_tan).
//   A_PHASE header of 1..16 other uncontrolled one-qubit ops on three local
//           bits, applied to registers in order (op_phase).
// A sweep that ends with a pass writes its results straight to memory and
// loads the next tile into the freed buffer meanwhile.
// Gradient terms: Re sum conj(lambda_k) (D_j psi_{k-1}) with psi_{k-1} = V psi_k,
// summed per thread, reduced per warp into shared slots [warp][slot], per CTA
// in warp order, and over CTAs in a fixed order by k_adj_slots: deterministic
// for a fixed grid.
#include <cuda_runtime.h>
#include <math.h>
#include <stddef.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "dq_adjsweep.cuh"
#include "dq_common.cuh"
#include "dq_engine.cuh"
#include "dq_gates.hpp"
#include "dq_handle.cuh"

namespace dq {
namespace {

constexpr int kAThreads = 256;
constexpr int kAWarps = kAThreads / 32;
constexpr uint32_t kAMaxLocal = 11;
constexpr uint32_t kALoMin = 3;  // qubits 0..2 stay local: 128-byte runs per tile load
constexpr uint32_t kAMaxOps = 192;
constexpr uint32_t kAMaxSlots = 192;

enum AType : uint8_t { A_ONE = 1, A_TWO = 2, A_DIAG = 3, A_PASS = 4, A_PHASE = 5 };
constexpr uint32_t kAPhaseOps = 16;  // ops of one register phase
constexpr uint32_t kAPhaseStage = 32;  // phase ops of a sweep staged once per CTA, at most
constexpr uint32_t kAMaxSweepOps = 2 * kAMaxOps;  // ops of a sweep, pass headers included
// shared memory of a sweep (bytes) up to which two CTAs share an SM; phase
// tables are staged while it is kept
constexpr size_t kATwoCtas = 108 * 1024;
constexpr uint32_t kATabTiles = 8;  // tiles of a state from which tables are staged

struct alignas(8) AOp {
  uint8_t type;
  uint8_t np;        // derivative matrices (gradient slots) of the op
  uint8_t lt, lt2;   // A_ONE: local target bit; A_TWO: local bits of the 4x4 MSB / LSB
  int8_t sel;        // A_ONE: non-local selector position (-1: none)
  uint8_t skip0;     // A_ONE with selector: variant 0 is the identity with no derivatives
  uint8_t dq[2];     // A_DIAG: qubit encodings (bit 7: local; low 7 bits: local bit or global position)
  uint8_t ndq;       // A_DIAG: 1 or 2 qubits (dq[0] = MSB of the diagonal index)
  uint8_t cnt;       // A_PASS, A_PHASE: number of one-qubit ops that follow it; A_ONE in one: 1 + its TanForm
  uint8_t pad[2];
  uint32_t lctrl;    // A_ONE: local control mask (tile offset bits), its TanForm record (pool offset);
                     // A_PASS, A_PHASE: its first PSub
  uint32_t slot;     // first sweep-local gradient slot; A_PASS: its diagonal run's record in the blob
  uint32_t mat;      // offset of the op's matrices in the pool (double2 units); A_PASS, A_PHASE:
                     // factor of both vectors after its ops (pool offset, kNone: 1)
};
// A_PASS, A_PHASE: lt, lt2, dq[0]: its register bits.  A_PASS: np: its diagonal
// run has gradient terms; ndq: it has a diagonal run; dq[1]: that run's index;
// pad[0]: its rotations' form (0: none)
constexpr uint32_t kNone = 0xffffffffu;
static_assert(sizeof(AOp) == 24 && offsetof(AOp, dq) == 6 && offsetof(AOp, ndq) == 8 && offsetof(AOp, lctrl) == 12,
              "AOp layout (passes read it as words)");

struct ASweepHdr {
  uint32_t n, m, nops, nslots;
  uint64_t ntiles;
  uint32_t lpos[kAMaxLocal];  // local bit positions, ascending
  uint32_t npos_cnt;
  uint32_t npos[64];          // non-local bit positions, ascending
  uint32_t phase_ops;         // > 0: every register phase's op data is staged once per CTA
                              // (pass header lctrl = its first PSub); 0: staged per tile
  uint32_t direct;            // the last op is a pass that writes to memory itself
  uint32_t blob0, nblob;      // diagonal runs' records: pool offset and length (double2 units)
  uint32_t ndrun, ntab;       // diagonal runs, and how many keep phase tables
};

// One sweep of one (psi, lambda) pair in a multi-job launch.
struct AJob {
  double2* psi;
  double2* lam;
  const ASweepHdr* hdr;
  const AOp* ops;
  const double2* pool;
  double* partial;       // [slot][chunk]
  const uint32_t* map;   // sweep-local slot -> index into out
  double* out;           // the pair's gradient slots
  uint32_t nslots, pad;
};

__device__ __forceinline__ double2 cfma2(double2 a, double2 b, double2 acc) {
  return make_double2(fma(a.x, b.x, fma(-a.y, b.y, acc.x)), fma(a.x, b.y, fma(a.y, b.x, acc.y)));
}
__device__ __forceinline__ double2 cmul2(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double redot(double2 l, double2 w, double acc) {
  return fma(l.x, w.x, fma(l.y, w.y, acc));
}
__device__ __forceinline__ uint32_t ins0a(uint32_t k, uint32_t p) {
  return ((k >> p) << (p + 1)) | (k & ((1u << p) - 1u));
}

// Shared-memory layout of a tile: element o lives at swz(o).  The low three
// index bits are XORed with a fold of the higher ones, so eight threads whose
// elements differ only in higher bits (register phases over low qubits,
// strided pairs) hit eight different 128-byte bank rows.  A bijection on
// [0, 2^m) for every m.
__device__ __forceinline__ uint32_t swz(uint32_t o) {
  return o ^ (((o >> 3) ^ (o >> 6) ^ (o >> 9)) & 7u);
}

__device__ __forceinline__ void cp_async16a(void* smem, const void* gmem) {
  const uint32_t sa = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}

// x[e] for a run-time e in 0..3 without indexing a local array
__device__ __forceinline__ double2 sel4(const double2 (&x)[4], uint32_t e) {
  const double2 lo = (e & 1u) ? x[1] : x[0];
  const double2 hi = (e & 1u) ? x[3] : x[2];
  return (e & 2u) ? hi : lo;
}

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

template <int NP>
__device__ __forceinline__ void flush_acc(const double (&acc)[4], double* accw, uint32_t slot) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    const double v = warp_sum_d(acc[j]);
    if (lane == 0) accw[slot + j] += v;
  }
}

template <int NP>
__device__ __noinline__ void op_one(double2* sp, double2* sl, const AOp& op, const double2* pool, uint32_t m,
                       uint64_t base, double* accw) {
  int var = 0;
  if (op.sel >= 0) var = (int)((base >> op.sel) & 1ULL);
  if (var == 0 && op.skip0) return;
  const double2* mt = pool + op.mat + (uint32_t)var * (4u + 4u * NP);
  double2 v[4], d[NP > 0 ? NP : 1][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = mt[i];
#pragma unroll
  for (int j = 0; j < NP; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) d[j][i] = mt[4 + 4 * j + i];
  // zero-insertion positions: target and local controls, ascending
  uint32_t pos[12];
  int npos = 0;
  uint32_t mask = op.lctrl | (1u << op.lt);
  while (mask) {
    const uint32_t b = __ffs(mask) - 1;
    pos[npos++] = b;
    mask &= mask - 1;
  }
  const uint32_t count = (1u << m) >> npos;
  const uint32_t tb = 1u << op.lt;
  const bool plain = op.lctrl == 0;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  for (uint32_t k = threadIdx.x; k < count; k += kAThreads) {
    uint32_t o;
    if (plain) {
      o = ins0a(k, op.lt);
    } else {
      o = k;
      for (int p = 0; p < npos; ++p) o = ins0a(o, pos[p]);
      o |= op.lctrl;
    }
    const uint32_t o1 = swz(o | tb);
    o = swz(o);
    const double2 a0 = sp[o], a1 = sp[o1], b0 = sl[o], b1 = sl[o1];
    const double2 p0 = cfma2(v[1], a1, cmul2(v[0], a0));
    const double2 p1 = cfma2(v[3], a1, cmul2(v[2], a0));
    sp[o] = p0;
    sp[o1] = p1;
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      const double2 w0 = cfma2(d[j][1], p1, cmul2(d[j][0], p0));
      const double2 w1 = cfma2(d[j][3], p1, cmul2(d[j][2], p0));
      acc[j] = redot(b0, w0, redot(b1, w1, acc[j]));
    }
    sl[o] = cfma2(v[1], b1, cmul2(v[0], b0));
    sl[o1] = cfma2(v[3], b1, cmul2(v[2], b0));
  }
  flush_acc<NP>(acc, accw, op.slot);
}

template <int NP>
__device__ __noinline__ void op_two(double2* sp, double2* sl, const AOp& op, const double2* pool, uint32_t m,
                       double* accw) {
  const double2* mt = pool + op.mat;
  const uint32_t ba = 1u << op.lt, bb = 1u << op.lt2;
  const uint32_t p0 = min((uint32_t)op.lt, (uint32_t)op.lt2), p1 = max((uint32_t)op.lt, (uint32_t)op.lt2);
  const uint32_t count = (1u << m) >> 2;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  for (uint32_t k = threadIdx.x; k < count; k += kAThreads) {
    const uint32_t b = ins0a(ins0a(k, p0), p1);
    const uint32_t idx[4] = {swz(b), swz(b | bb), swz(b | ba), swz(b | ba | bb)};
    double2 x[4], y[4], p[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      x[r] = sp[idx[r]];
      y[r] = sl[idx[r]];
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      double2 s = make_double2(0.0, 0.0);
#pragma unroll
      for (int c = 0; c < 4; ++c) s = cfma2(mt[r * 4 + c], x[c], s);
      p[r] = s;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      sp[idx[r]] = p[r];
      double2 s = make_double2(0.0, 0.0);
#pragma unroll
      for (int c = 0; c < 4; ++c) s = cfma2(mt[r * 4 + c], y[c], s);
#pragma unroll
      for (int j = 0; j < NP; ++j) {
        double2 w = make_double2(0.0, 0.0);
#pragma unroll
        for (int c = 0; c < 4; ++c) w = cfma2(mt[16 * (j + 1) + r * 4 + c], p[c], w);
        acc[j] = redot(y[r], w, acc[j]);
      }
      sl[idx[r]] = s;
    }
  }
  flush_acc<NP>(acc, accw, op.slot);
}

template <int NP>
__device__ __noinline__ void op_diag(double2* sp, double2* sl, const AOp& op, const double2* pool, uint32_t m,
                        uint64_t base, double* accw) {
  // entry index bits: for each diag qubit, its bit from the tile offset (local)
  // or from the tile base (non-local)
  const double2* mt = pool + op.mat;  // [4 entries: v], then [NP][4]: d
  uint32_t lmask[2] = {0, 0}, fixed = 0;
  for (uint32_t a = 0; a < op.ndq; ++a) {
    const uint32_t e = op.dq[a];
    const uint32_t shift = op.ndq - 1 - a;  // dq[0] is the MSB
    if (e & 0x80u) lmask[a] = 1u << (e & 0x7fu);
    else fixed |= (uint32_t)((base >> (e & 0x7fu)) & 1ULL) << shift;
  }
  double2 v[4], d[NP > 0 ? NP : 1][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = mt[i];
#pragma unroll
  for (int j = 0; j < NP; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) d[j][i] = mt[4 + 4 * j + i];
  const uint32_t L = 1u << m;
  const uint32_t sh0 = op.ndq == 2 ? 1u : 0u;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  for (uint32_t o = threadIdx.x; o < L; o += kAThreads) {
    uint32_t e = fixed;
    if (lmask[0] && (o & lmask[0])) e |= 1u << sh0;
    if (lmask[1] && (o & lmask[1])) e |= 1u;
    const uint32_t so = swz(o);
    const double2 a = sp[so], b = sl[so];
    const double2 ve = sel4(v, e);
    const double2 p = cmul2(ve, a);
    sp[so] = p;
#pragma unroll
    for (int j = 0; j < NP; ++j) acc[j] = redot(b, cmul2(sel4(d[j], e), p), acc[j]);
    sl[so] = cmul2(ve, b);
  }
  flush_acc<NP>(acc, accw, op.slot);
}

// ---- runs of diagonal gates ----
//
// Every diagonal gate is exp(i theta(b0, b1)), so a run of them is one phase
// exp(i Theta(x)) with Theta a quadratic polynomial in the index bits.  Each
// bit is a register bit of the pass, a bit of threadIdx.x or a bit of the
// tile's base.  Theta splits into
//   - local linear and quadratic terms: per thread a factor and one factor per
//     register bit (pair_factors), the same for every tile: kept in a table in
//     shared memory where there are tiles and room enough;
//   - terms with base bits: a constant and a factor per coupled local bit,
//     a dozen numbers a tile, made by one warp while the tile is loaded.
// An element's phase is a product of these: 4 sincos a thread and tile without
// the table and none with it, where a sincos per element of a summed angle
// took 8 (and rounded the sum of all angles).
//
// Gradients.  The entries have modulus one, so conj(lambda) psi is the same
// before every gate of the run, and dU U^dagger = i g with g real: a term is a
// sum of at most four Walsh coefficients of z = Im(conj(lambda) psi), its g in
// the Walsh basis of its two bits.  A warp transforms its 256 values over the
// three register bits and the five lane bits (each lane bit is first exchanged
// with a register bit: 40 shuffles a thread against 160 for butterflies on the
// complex product), then lane j adds term j to its warp's slot.
struct DTerm {
  double w;
  uint32_t code;  // source lane : 5, warp bits : 3, register : 3, two base bits : 6 each (63: none),
                  // registers that its 32 terms use : 8
  uint32_t slot;
};
struct DAng {
  double ang;
  uint32_t code;
  uint32_t pad;
};
// A run's record in the blob (double2 units): 0: (constant angle, factor of
// both vectors); 1..3: exp(i H01), exp(i H02), exp(i H12) of the register
// pairs; 4: counts; 5: masks and table; then its terms and angle lists.
struct DCount {
  uint32_t nterm;
  uint32_t ends;   // local angles: cumulative ends of the lists of T, G0, G1, G2 (a byte each)
  uint32_t ncst, nlin;
};
struct DMask {
  uint32_t coupled;  // thread bits 0..7, register bits 8..10 with terms in base bits
  uint32_t pairs;    // register pairs 01, 02, 12 with a term
  uint32_t tab;
  uint32_t layers;   // its terms in up to four lists (a byte each) with one term of a gate each
};
constexpr uint32_t kDRunHdr = 6, kDFactors = 12;

__device__ __forceinline__ double2 expi(double a) {
  double sn, cs;
  sincos(a, &sn, &cs);
  return make_double2(cs, sn);
}

__device__ __forceinline__ void pair_factors(const double2* B, double2 (&f)[4]) {
  const DCount& C = *reinterpret_cast<const DCount*>(B + 4);
  const DAng* L = reinterpret_cast<const DAng*>(B + kDRunHdr + C.nterm);
  uint32_t j = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint32_t e = (C.ends >> (8 * k)) & 0xffu;
    double x = 0.0;
    for (; j < e; ++j)
      if ((threadIdx.x & L[j].code) == L[j].code) x += L[j].ang;
    f[k] = expi(x);
  }
}

// The factors of a run that depend on the tile: E[0..10] per local bit code,
// E[11] the constant (one warp).
__device__ __forceinline__ void tile_factors(const double2* B, uint64_t base, double2* E) {
  const uint32_t lane = threadIdx.x & 31;
  const DCount& C = *reinterpret_cast<const DCount*>(B + 4);
  const DAng* cst = reinterpret_cast<const DAng*>(B + kDRunHdr + C.nterm + (C.ends >> 24));
  const DAng* lin = cst + C.ncst;
  double c = 0.0;
  for (uint32_t j = lane; j < C.ncst; j += 32) {
    const uint32_t p = cst[j].code & 63u, q = (cst[j].code >> 6) & 63u;
    if ((base >> p & 1ULL) && (q == 63u || (base >> q & 1ULL))) c += cst[j].ang;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  double x = lane == 11 ? B[0].x + c : 0.0;
  for (uint32_t j = 0; j < C.nlin; ++j)
    if ((lin[j].code & 15u) == lane && (base >> (lin[j].code >> 4) & 1ULL)) x += lin[j].ang;
  if (lane < kDFactors) {
    double2 e = expi(x);
    if (lane == 11) e = make_double2(e.x * B[0].y, e.y * B[0].y);
    E[lane] = e;
  }
}

// Exchanges register bit KB with lane bit LB, then the butterfly on it.
template <int KB, int LB>
__device__ __forceinline__ void walsh_lane(double (&z)[8], int lane) {
  const bool up = (lane >> LB) & 1;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (!(i >> KB & 1)) {
      const int k = i | (1 << KB);
      const double r = __shfl_xor_sync(0xffffffffu, up ? z[i] : z[k], 1 << LB);
      const double kept = up ? z[k] : z[i], d = kept - r;
      z[i] = kept + r;
      z[k] = up ? -d : d;
    }
}

__device__ __forceinline__ void diag_grads(const double2 (&a)[8], const double2 (&b)[8], const double2* B,
                                           uint64_t base, bool valid, double* accw) {
  const int lane = threadIdx.x & 31;
  const uint32_t w = threadIdx.x >> 5;
  const uint32_t layers = reinterpret_cast<const DMask*>(B + 5)->layers;
  const DTerm* terms = reinterpret_cast<const DTerm*>(B + kDRunHdr);
  double z[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) z[i] = valid ? fma(b[i].x, a[i].y, -b[i].y * a[i].x) : 0.0;
#pragma unroll
  for (int s = 1; s < 8; s <<= 1)
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (!(i & s)) {
        const double u = z[i], v = z[i | s];
        z[i] = u + v;
        z[i | s] = u - v;
      }
  walsh_lane<0, 0>(z, lane);
  walsh_lane<1, 1>(z, lane);
  walsh_lane<2, 2>(z, lane);
  walsh_lane<0, 3>(z, lane);
  walsh_lane<1, 4>(z, lane);
  // the coefficient of register mask R, lane mask M is now in lane
  // R | (M & 3) << 3, register M3 | M4 << 1 | M2 << 2
  for (uint32_t left = layers; left; left >>= 8) {
    const uint32_t cnt = left & 0xffu;
    for (uint32_t c0 = 0; c0 < cnt; c0 += 32) {
      const DTerm t = terms[min(c0 + (uint32_t)lane, cnt - 1u)];
      const uint32_t used = t.code >> 23, reg = (t.code >> 8) & 7u;
      double v = 0.0;
#pragma unroll
      for (uint32_t r = 0; r < 8; ++r)
        if (used >> r & 1u) {
          const double x = __shfl_sync(0xffffffffu, z[r], (int)(t.code & 31u));
          if (reg == r) v = x;
        }
      const uint32_t p = (t.code >> 11) & 63u, q = (t.code >> 17) & 63u;
      const uint32_t neg = __popc((t.code >> 5) & w & 7u) + (p != 63u ? (uint32_t)(base >> p) & 1u : 0u) +
                           (q != 63u ? (uint32_t)(base >> q) & 1u : 0u);
      if (c0 + (uint32_t)lane < cnt) accw[t.slot] += (neg & 1u) ? -t.w * v : t.w * v;
    }
    terms += cnt;
    __syncwarp();  // another lane may add to the same slot in the next list
  }
}

__device__ __forceinline__ void diag_apply(double2 (&a)[8], double2 (&b)[8], const double2* B, const double2* E,
                                           const double2* tabs) {
  const DMask M = *reinterpret_cast<const DMask*>(B + 5);
  double2 f[4];
  if (M.tab != kNone) {
    const double2* tb = tabs + (size_t)M.tab * 4 * kAThreads + threadIdx.x;
#pragma unroll
    for (int k = 0; k < 4; ++k) f[k] = tb[k * kAThreads];
  } else {
    pair_factors(B, f);
  }
  f[0] = cmul2(f[0], E[11]);
#pragma unroll 1
  for (uint32_t c = M.coupled & 0xffu; c; c &= c - 1) {
    const uint32_t r = __ffs(c) - 1;
    if (threadIdx.x >> r & 1u) f[0] = cmul2(f[0], E[r]);
  }
#pragma unroll
  for (int k = 0; k < 3; ++k)
    if (M.coupled >> (8 + k) & 1u) f[k + 1] = cmul2(f[k + 1], E[8 + k]);
  double2 h[4] = {f[0], cmul2(f[0], f[1]), cmul2(f[0], f[2]), make_double2(0.0, 0.0)};
  h[3] = cmul2(h[1], f[2]);
  if (M.pairs & 1u) h[3] = cmul2(h[3], B[1]);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    a[i] = cmul2(h[i], a[i]);
    b[i] = cmul2(h[i], b[i]);
    double2 g = cmul2(h[i], f[3]);
    if ((i & 1) && (M.pairs & 2u)) g = cmul2(g, B[2]);
    if ((i & 2) && (M.pairs & 4u)) g = cmul2(g, B[3]);
    a[i | 4] = cmul2(g, a[i | 4]);
    b[i | 4] = cmul2(g, b[i | 4]);
  }
}

// One op of a register phase staged in shared memory.
struct PSub {
  double2 v[4];      // U^dagger
  double2 d[4][4];   // np derivatives in the form D' = dU U^dagger (applied to psi before V)
  uint32_t pb;       // index of the target among the phase bits
  uint32_t vk;       // 0: general V; 1: real V; 2: real diagonal, imaginary off-diagonal;
                     // 3 + TanForm: v[0] = (t, gradient weight)
  uint32_t np, slot;
  uint32_t tm[4];    // per derivative: bit 2e / 2e + 1 set if Re / Im of D'[e] is non-zero
};

template <int PB>
__device__ __forceinline__ int pair_lo(int k) {  // k-th index with bit PB clear
  return PB == 0 ? 2 * k : (PB == 1 ? (k & 1) | ((k & 2) << 1) : k);
}

// Re sum over the thread's pairs of conj(lambda) D' psi, term by term of D':
// Re(D'[r][c] conj(l_r) p_c) = Re D' Re(conj(l_r) p_c) - Im D' Im(conj(l_r) p_c),
// skipping the parts of D' that are zero (ry: two real entries, rx: two
// imaginary ones).
template <int PB>
__device__ __forceinline__ double grad_terms(const double2 (&a)[8], const double2 (&b)[8], const double2* dp,
                                             uint32_t tm) {
  double s = 0.0;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int r = e >> 1, c = e & 1;
    if (tm & (1u << (2 * e))) {
      double t[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int i = pair_lo<PB>(k), j = i | (1 << PB);
        const double2 l = b[r ? j : i], p = a[c ? j : i];
        t[k] = fma(l.x, p.x, l.y * p.y);
      }
      s = fma(dp[e].x, (t[0] + t[1]) + (t[2] + t[3]), s);
    }
    if (tm & (2u << (2 * e))) {
      double t[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int i = pair_lo<PB>(k), j = i | (1 << PB);
        const double2 l = b[r ? j : i], p = a[c ? j : i];
        t[k] = fma(l.x, p.y, -l.y * p.x);
      }
      s = fma(-dp[e].y, (t[0] + t[1]) + (t[2] + t[3]), s);
    }
  }
  return s;
}

// y = V x on one pair for the three shapes of V
template <int VK>
__device__ __forceinline__ void apply2(const double2* v, double2& x0, double2& x1) {
  const double2 a0 = x0, a1 = x1;
  if (VK == 1) {
    x0 = make_double2(fma(v[1].x, a1.x, v[0].x * a0.x), fma(v[1].x, a1.y, v[0].x * a0.y));
    x1 = make_double2(fma(v[3].x, a1.x, v[2].x * a0.x), fma(v[3].x, a1.y, v[2].x * a0.y));
  } else if (VK == 2) {
    x0 = make_double2(fma(-v[1].y, a1.y, v[0].x * a0.x), fma(v[1].y, a1.x, v[0].x * a0.y));
    x1 = make_double2(fma(v[3].x, a1.x, -v[2].y * a0.y), fma(v[3].x, a1.y, v[2].y * a0.x));
  } else {
    x0 = cfma2(v[1], a1, cmul2(v[0], a0));
    x1 = cfma2(v[3], a1, cmul2(v[2], a0));
  }
}

template <int PB, int VK>
__device__ __forceinline__ void phase_one(double2 (&a)[8], double2 (&b)[8], const PSub& P,
                                          double (&acc)[4]) {
  // gradient terms Re <lambda_k| dU U^dagger |psi_k> from the amplitudes
  // before the op, then psi and lambda both take V = U^dagger
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (q < (int)P.np) acc[q] = grad_terms<PB>(a, b, P.d[q], P.tm[q]);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int i = pair_lo<PB>(k), j = i | (1 << PB);
    apply2<VK>(P.v, a[i], a[j]);
    apply2<VK>(P.v, b[i], b[j]);
  }
}

// A rotation about Y or X undone up to its scale: V = cos (I + tan G); the host
// collects the cosines (one factor a sweep) and weights the gradient term with
// what was not yet applied.  4 FMA a pair and vector against 8, and 4 for the
// gradient term sum conj(lambda) G psi of the generator G.
enum TanForm : uint32_t { TF_Y = 0, TF_X = 1 };

template <int PB, uint32_t TF>
__device__ __forceinline__ double tan_op(double2 (&a)[8], double2 (&b)[8], double t) {
  double s[2] = {0.0, 0.0};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int i = pair_lo<PB>(k), j = i | (1 << PB);
    const double2 l0 = b[i], l1 = b[j], p0 = a[i], p1 = a[j];
    double& x = s[k & 1];
    if (TF == TF_Y) {
      x = fma(l1.x, p0.x, fma(l1.y, p0.y, fma(-l0.x, p1.x, fma(-l0.y, p1.y, x))));
      a[i] = make_double2(fma(t, p1.x, p0.x), fma(t, p1.y, p0.y));
      a[j] = make_double2(fma(-t, p0.x, p1.x), fma(-t, p0.y, p1.y));
      b[i] = make_double2(fma(t, l1.x, l0.x), fma(t, l1.y, l0.y));
      b[j] = make_double2(fma(-t, l0.x, l1.x), fma(-t, l0.y, l1.y));
    } else {
      x = fma(l0.x, p1.y, fma(-l0.y, p1.x, fma(l1.x, p0.y, fma(-l1.y, p0.x, x))));
      a[i] = make_double2(fma(-t, p1.y, p0.x), fma(t, p1.x, p0.y));
      a[j] = make_double2(fma(-t, p0.y, p1.x), fma(t, p0.x, p1.y));
      b[i] = make_double2(fma(-t, l1.y, l0.x), fma(t, l1.x, l0.y));
      b[j] = make_double2(fma(-t, l0.y, l1.x), fma(t, l0.x, l1.y));
    }
  }
  return s[0] + s[1];
}

template <int PB>
__device__ __forceinline__ void general_op(double2 (&a)[8], double2 (&b)[8], const PSub& P, bool valid,
                                           double* accw) {
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  if (P.vk == 0) phase_one<PB, 0>(a, b, P, acc);
  else if (P.vk == 1) phase_one<PB, 1>(a, b, P, acc);
  else phase_one<PB, 2>(a, b, P, acc);
#pragma unroll
  for (uint32_t q = 0; q < 4; ++q) {
    if (q >= P.np) break;
    const double v = warp_sum_d(valid ? acc[q] : 0.0);
    if ((threadIdx.x & 31) == 0) accw[P.slot + q] += v;
  }
}

// Sums of four values over the warp: lane l < 4 returns the sum of g[l] (12
// shuffles against 40 for one after the other).
__device__ __forceinline__ double warp_sum4(const double (&g)[4]) {
  const int lane = threadIdx.x & 31;
  const bool b0 = lane & 1, b1 = lane & 2;
  const double x = (b0 ? g[1] : g[0]) + __shfl_xor_sync(0xffffffffu, b0 ? g[0] : g[1], 1);
  const double y = (b0 ? g[3] : g[2]) + __shfl_xor_sync(0xffffffffu, b0 ? g[2] : g[3], 1);
  double v = (b1 ? y : x) + __shfl_xor_sync(0xffffffffu, b1 ? x : y, 2);
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// N rotations of one form on register bits 0 .. N - 1 (the passes of layered
// circuits), without a branch between them.
template <uint32_t TF, int N>
__device__ __forceinline__ void pass_tan(double2 (&a)[8], double2 (&b)[8], const PSub* ps, bool valid,
                                         double* accw) {
  double g[4] = {0.0, 0.0, 0.0, 0.0};
  g[0] = tan_op<0, TF>(a, b, ps[0].v[0].x);
  if constexpr (N > 1) g[1] = tan_op<1, TF>(a, b, ps[1].v[0].x);
  if constexpr (N > 2) g[2] = tan_op<2, TF>(a, b, ps[2].v[0].x);
#pragma unroll
  for (int k = 0; k < N; ++k) g[k] = valid ? g[k] : 0.0;
  const double v = warp_sum4(g);
  const uint32_t lane = threadIdx.x & 31;
  if (lane < N && ps[lane].np) accw[ps[lane].slot] += ps[lane].v[0].y * v;
}

// The op data of one register phase: threads th < cnt fill ps[0 .. cnt).
__device__ __forceinline__ void stage_phase(const AOp& hdr, const AOp* sub, const double2* pool,
                                            PSub* ps, uint32_t th) {
  const uint32_t cnt = hdr.cnt;
  const uint32_t pbits[3] = {hdr.lt, hdr.lt2, (uint32_t)hdr.dq[0]};
  if (th < cnt) {
    const AOp op = sub[th];
    PSub& P = ps[th];
    const double2* mt = pool + op.mat;
    P.np = op.np;
    P.slot = op.slot;
    P.pb = op.lt == pbits[0] ? 0u : (op.lt == pbits[1] ? 1u : 2u);
    if (op.cnt) {
      P.vk = 2u + op.cnt;
      P.v[0] = pool[op.lctrl];
      return;
    }
    for (int i = 0; i < 4; ++i) P.v[i] = mt[i];
    const bool real = mt[0].y == 0.0 && mt[1].y == 0.0 && mt[2].y == 0.0 && mt[3].y == 0.0;
    const bool rxl = mt[0].y == 0.0 && mt[3].y == 0.0 && mt[1].x == 0.0 && mt[2].x == 0.0;
    P.vk = real ? 1u : (rxl ? 2u : 0u);
    // D' blocks follow the dU blocks (uncontrolled one-qubit ops only)
    for (uint32_t q = 0; q < op.np; ++q) {
      uint32_t tm = 0;
      for (int i = 0; i < 4; ++i) {
        const double2 dv = mt[4 + 4 * op.np + 4 * q + i];
        P.d[q][i] = dv;
        tm |= (dv.x != 0.0 ? 1u : 0u) << (2 * i);
        tm |= (dv.y != 0.0 ? 2u : 0u) << (2 * i);
      }
      P.tm[q] = tm;
    }
  }
}

// The register layout of a pass or phase on local bits q0, q1, q2: thread g
// holds the elements ob | bits (in the tile at off(e)).
struct RegBits {
  uint32_t ob, sb, s0, s1, s2;
  __device__ __forceinline__ RegBits(uint32_t q0, uint32_t q1, uint32_t q2, uint32_t groups) {
    const uint32_t lo = min(q0, min(q1, q2)), hi = max(q0, max(q1, q2)), mid = q0 + q1 + q2 - lo - hi;
    ob = ins0a(ins0a(ins0a(threadIdx.x & (groups - 1u), lo), mid), hi);
    // swz is linear over XOR and ob has the three bits clear, so
    // swz(ob | bits) = swz(ob) ^ swz(bits)
    sb = swz(ob);
    s0 = swz(1u << q0);
    s1 = swz(1u << q1);
    s2 = swz(1u << q2);
  }
  __device__ __forceinline__ uint32_t off(int e) const {
    return sb ^ ((e & 1) ? s0 : 0u) ^ ((e & 2) ? s1 : 0u) ^ ((e & 4) ? s2 : 0u);
  }
};

__device__ __forceinline__ void scale8(double2 (&a)[8], double f) {
#pragma unroll
  for (int e = 0; e < 8; ++e) a[e] = make_double2(f * a[e].x, f * a[e].y);
}

// A register phase of any uncontrolled one-qubit ops, in order.  The gradient
// sums of up to four rotations are reduced together.
__device__ __noinline__ void op_phase(double2* sp, double2* sl, const AOp& hdr, const PSub* ps,
                                      const double2* pool, uint32_t m, double* accw) {
  const uint32_t lane = threadIdx.x & 31, groups = (1u << m) >> 3;
  const bool valid = threadIdx.x < groups;
  const RegBits rb(hdr.lt, hdr.lt2, hdr.dq[0], groups);
  double2 a[8], b[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    a[e] = sp[rb.off(e)];
    b[e] = sl[rb.off(e)];
  }
  double g[4] = {0.0, 0.0, 0.0, 0.0};
  uint32_t who = 0, pending = 0;  // the ops of g, a byte each
  auto flush = [&]() {
    const double v = warp_sum4(g);
    if (lane < pending) {
      const PSub& P = ps[(who >> (8 * lane)) & 0xffu];
      if (P.np) accw[P.slot] += P.v[0].y * v;
    }
    pending = 0;
  };
#pragma unroll 1
  for (uint32_t u = 0; u < hdr.cnt; ++u) {
    const PSub& P = ps[u];
    const double t = P.v[0].x;
    double v = 0.0;
    switch (P.pb * 8 + P.vk) {
      case 3: v = tan_op<0, TF_Y>(a, b, t); break;
      case 4: v = tan_op<0, TF_X>(a, b, t); break;
      case 11: v = tan_op<1, TF_Y>(a, b, t); break;
      case 12: v = tan_op<1, TF_X>(a, b, t); break;
      case 19: v = tan_op<2, TF_Y>(a, b, t); break;
      case 20: v = tan_op<2, TF_X>(a, b, t); break;
      default:
        if (P.pb == 0) general_op<0>(a, b, P, valid, accw);
        else if (P.pb == 1) general_op<1>(a, b, P, valid, accw);
        else general_op<2>(a, b, P, valid, accw);
        continue;
    }
    if (pending == 4) flush();
    g[3] = g[2];
    g[2] = g[1];
    g[1] = g[0];
    g[0] = valid ? v : 0.0;
    who = who << 8 | u;
    ++pending;
  }
  if (pending) flush();
  if (hdr.mat != kNone) {
    scale8(a, pool[hdr.mat].x);
    scale8(b, pool[hdr.mat].x);
  }
  if (valid) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      sp[rb.off(e)] = a[e];
      sl[rb.off(e)] = b[e];
    }
  }
}

// One backward sweep over tiles t0, t0 + step, ... (< t1) of psi and lambda;
// the CTA's gradient sums go to partial[slot * nparts + part].  Every thread
// of the CTA calls it; the caller separates consecutive calls by a barrier.
// The pass that ends a sweep holds the whole tile in registers: the next
// tile's copies start before its arithmetic, and its results go to memory from
// the registers (each eight threads 128 consecutive bytes).
// 24 qubits, 16 layers of ry, rz and rzz: 42 sweeps in 14.1 ms, of which 8.6 are
// the tiles' loads and stores alone (1.07 GB a sweep at 5.2 TB/s), 2.0 the passes
// through shared memory and 3.6 arithmetic that does not hide behind them; 24.3 ms
// with separate passes for runs and rotations, general 2x2s, a warp sum a rotation
// and loads that began after the stores.  128 such sets of 20 qubits and 8
// layers: 53 ms, 93 before.  Prefetching the next tile into L2 at the start of
// this one gains nothing.
__device__ __forceinline__ void adj_sweep_body(double2* __restrict__ psi, double2* __restrict__ lam,
                                               const ASweepHdr* __restrict__ hp,
                                               const AOp* __restrict__ ops,
                                               const double2* __restrict__ pool, double* partial,
                                               uint32_t part, uint32_t nparts, uint64_t t0,
                                               uint64_t t1, uint64_t step) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ ASweepHdr H;
  __shared__ uint64_t hi_tab[1u << (kAMaxLocal - kALoMin)];
  if (threadIdx.x == 0) H = *hp;
  __syncthreads();
  const uint32_t m = H.m, L = 1u << m;
  const uint32_t w = threadIdx.x >> 5;
  double2* sp = reinterpret_cast<double2*>(smraw);
  double2* sl = sp + L;
  double2* tabs = sl + L;
  double2* blob = tabs + (size_t)H.ntab * 4 * kAThreads;
  double2* fact = blob + H.nblob;  // [tile parity][run][kDFactors]
  double* acc0 = reinterpret_cast<double*>(fact + 2 * kDFactors * H.ndrun);
  double* accw = acc0 + w * H.nslots;
  // the sweep's ops, and (phase_ops > 0) every pass's op data, in shared
  // memory for the whole launch
  AOp* sops = reinterpret_cast<AOp*>(acc0 + (H.nslots ? H.nslots : 1u) * kAWarps);
  PSub* psall = reinterpret_cast<PSub*>(sops + (H.nops + 1u) / 2u * 2u);
  for (uint32_t i = threadIdx.x; i < H.nslots * kAWarps; i += kAThreads) acc0[i] = 0.0;
  for (uint32_t i = threadIdx.x; i < H.nops; i += kAThreads) sops[i] = ops[i];
  for (uint32_t i = threadIdx.x; i < H.nblob; i += kAThreads) blob[i] = pool[H.blob0 + i];
  // offset bits above the 5 contiguous ones -> global bits
  // local bits 0 .. lo_bits-1 are qubits 0 .. lo_bits-1: runs of 2^lo_bits
  // consecutive amplitudes (at least 128 B)
  uint32_t lo_bits = 0;
  while (lo_bits < m && lo_bits < 5 && H.lpos[lo_bits] == lo_bits) ++lo_bits;
  const uint32_t nhi = m - lo_bits;
  for (uint32_t hv = threadIdx.x; hv < (1u << nhi); hv += kAThreads) {
    uint64_t g = 0;
    for (uint32_t b = 0; b < nhi; ++b)
      if (hv >> b & 1u) g |= 1ULL << H.lpos[lo_bits + b];
    hi_tab[hv] = g;
  }
  __syncthreads();
  // a pass per warp: their loads from memory side by side (u3 on 14 qubits: 11 sweeps
  // in 0.46 ms, 0.47 with one pass after the other)
  for (uint32_t i = 0, k = 0; i < H.nops; ++i) {
    const AOp op = sops[i];
    if (op.type != A_PASS && op.type != A_PHASE) continue;
    if (H.phase_ops && (k++ & (kAWarps - 1)) == w)
      stage_phase(op, sops + i + 1, pool, psall + op.lctrl, threadIdx.x & 31u);
    if (op.type == A_PASS && op.ndq) {
      const double2* B = blob + op.slot;
      const uint32_t tab = reinterpret_cast<const DMask*>(B + 5)->tab;
      if (tab != kNone) {
        double2 f[4];
        pair_factors(B, f);
#pragma unroll
        for (int k = 0; k < 4; ++k) tabs[((size_t)tab * 4 + k) * kAThreads + threadIdx.x] = f[k];
      }
    }
    i += op.cnt;
  }
  const uint32_t lo_mask = (1u << lo_bits) - 1u;
  // tile index -> its base (the index's bits on the non-local qubits), and the
  // base of a tile `step` further on: with ones in the local bits a carry
  // passes over them
  auto deposit = [&](uint64_t t) {
    uint64_t base = 0;
    for (uint32_t b = 0; b < H.npos_cnt; ++b)
      if (t >> b & 1ULL) base |= 1ULL << H.npos[b];
    return base;
  };
  uint64_t local = 0;
  for (uint32_t b = 0; b < m; ++b) local |= 1ULL << H.lpos[b];
  const uint64_t advance = deposit(step);
  // all of a tile's copies in flight at once (cp.async straight into the
  // swizzled layout)
  const uint32_t my_s = swz(threadIdx.x & (L - 1u));
  const uint64_t my_g = (threadIdx.x & lo_mask) | hi_tab[(threadIdx.x & (L - 1u)) >> lo_bits];
  auto load_tile = [&](uint64_t base) {
    if (m == kAMaxLocal) {
      const uint64_t h0 = 1ULL << H.lpos[8], h1 = 1ULL << H.lpos[9], h2 = 1ULL << H.lpos[10];
      const double2 *gp = psi + (base | my_g), *gl = lam + (base | my_g);
#pragma unroll
      for (uint32_t j = 0; j < 8; ++j) {
        const uint64_t g = ((j & 1u) ? h0 : 0ULL) + ((j & 2u) ? h1 : 0ULL) + ((j & 4u) ? h2 : 0ULL);
        const uint32_t o = my_s ^ swz(j * kAThreads);
        cp_async16a(sp + o, gp + g);
        cp_async16a(sl + o, gl + g);
      }
    } else {
      for (uint32_t o = threadIdx.x; o < L; o += kAThreads) {
        const uint64_t g = base | (o & lo_mask) | hi_tab[o >> lo_bits];
        cp_async16a(sp + swz(o), psi + g);
        cp_async16a(sl + swz(o), lam + g);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };

  bool loaded = false;
  uint32_t parity = 0;
  uint64_t base = deposit(t0), next = 0;
  const uint64_t tend = t1 < H.ntiles ? t1 : H.ntiles;
  for (uint64_t t = t0; t < tend; t += step, parity ^= 1u, base = next) {
    next = ((base | local) + advance) & ~local;
    if (!loaded) load_tile(base);
    loaded = false;
    // (the other parity's factors may still be in use)
    double2* E = fact + parity * kDFactors * H.ndrun;
    {
      const uint32_t* off = reinterpret_cast<const uint32_t*>(blob);
      for (uint32_t d = w; d < H.ndrun; d += kAWarps) tile_factors(blob + off[d], base, E + kDFactors * d);
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    for (uint32_t i = 0; i < H.nops; ++i) {
      const uint2* ow = reinterpret_cast<const uint2*>(sops + i);
      const uint2 w0 = ow[0];
      if ((w0.x & 0xffu) >= A_PASS) {
        const uint2 w1 = ow[1], w2 = ow[2];
        const uint32_t cnt = (w1.x >> 8) & 0xffu;
        const PSub* ps = psall + (H.phase_ops ? w1.y : 0u);
        if (!H.phase_ops && cnt) {
          stage_phase(sops[i], sops + i + 1, pool, psall, threadIdx.x);
          __syncthreads();
        }
        if ((w0.x & 0xffu) == A_PHASE) {
          op_phase(sp, sl, sops[i], ps, pool, m, accw);
          i += cnt;
          __syncthreads();
          continue;
        }
        const uint32_t q0 = (w0.x >> 16) & 0xffu, q1 = w0.x >> 24, q2 = (w0.y >> 16) & 0xffu;
        const bool valid = threadIdx.x < (L >> 3);
        const RegBits rb(q0, q1, q2, L >> 3);
        double2 a[8], b[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          a[e] = sp[rb.off(e)];
          b[e] = sl[rb.off(e)];
        }
        i += cnt;
        const bool direct = H.direct && i + 1 == H.nops;
        if (direct) {
          __syncthreads();
          if (t + step < tend) {
            load_tile(next);
            loaded = true;
          }
        }
        if (w1.x & 0xffu) {
          const double2* B = blob + w2.x;
          if (w0.x & 0xff00u) diag_grads(a, b, B, base, valid, accw);
          diag_apply(a, b, B, E + kDFactors * (w0.y >> 24), tabs);
        }
        switch ((w1.x >> 16) & 0xffu) {  // AOp::pad[0]: 1 + TanForm + 2 (count - 1)
          case 1: pass_tan<TF_Y, 1>(a, b, ps, valid, accw); break;
          case 2: pass_tan<TF_X, 1>(a, b, ps, valid, accw); break;
          case 3: pass_tan<TF_Y, 2>(a, b, ps, valid, accw); break;
          case 4: pass_tan<TF_X, 2>(a, b, ps, valid, accw); break;
          case 5: pass_tan<TF_Y, 3>(a, b, ps, valid, accw); break;
          case 6: pass_tan<TF_X, 3>(a, b, ps, valid, accw); break;
          default: break;
        }
        if (w2.y != kNone) {
          const double f = __ldg(&pool[w2.y].x);
          scale8(a, f);
          scale8(b, f);
        }
        if (direct) {
          const uint64_t gb = base | (rb.ob & lo_mask) | hi_tab[rb.ob >> lo_bits];
          const uint64_t g0 = 1ULL << H.lpos[q0], g1 = 1ULL << H.lpos[q1], g2 = 1ULL << H.lpos[q2];
          if (valid) {
            double2 *gp = psi + gb, *gl = lam + gb;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const uint64_t g = ((e & 1) ? g0 : 0ULL) + ((e & 2) ? g1 : 0ULL) + ((e & 4) ? g2 : 0ULL);
              gp[g] = a[e];
              gl[g] = b[e];
            }
          }
          break;
        }
        if (valid) {
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            sp[rb.off(e)] = a[e];
            sl[rb.off(e)] = b[e];
          }
        }
        __syncthreads();
        continue;
      }
      const AOp op = sops[i];
      switch (op.type) {
        case A_ONE:
          switch (op.np) {
            case 0: op_one<0>(sp, sl, op, pool, m, base, accw); break;
            case 1: op_one<1>(sp, sl, op, pool, m, base, accw); break;
            case 2: op_one<2>(sp, sl, op, pool, m, base, accw); break;
            case 3: op_one<3>(sp, sl, op, pool, m, base, accw); break;
            default: op_one<4>(sp, sl, op, pool, m, base, accw); break;
          }
          break;
        case A_TWO:
          if (op.np) op_two<1>(sp, sl, op, pool, m, accw);
          else op_two<0>(sp, sl, op, pool, m, accw);
          break;
        default:
          if (op.np) op_diag<1>(sp, sl, op, pool, m, base, accw);
          else op_diag<0>(sp, sl, op, pool, m, base, accw);
          break;
      }
      __syncthreads();
    }
    if (!H.direct) {
      for (uint32_t o = threadIdx.x; o < L; o += kAThreads) {
        const uint64_t g = base | (o & lo_mask) | hi_tab[o >> lo_bits];
        psi[g] = sp[swz(o)];
        lam[g] = sl[swz(o)];
      }
      __syncthreads();
    }
  }
  __syncthreads();
  for (uint32_t s = threadIdx.x; s < H.nslots; s += kAThreads) {
    double x = 0.0;
    for (int v = 0; v < kAWarps; ++v) x += acc0[v * H.nslots + s];
    partial[(size_t)s * nparts + part] = x;
  }
}

__global__ void __launch_bounds__(kAThreads, 2)
    k_adj_sweep(double2* __restrict__ psi, double2* __restrict__ lam, const ASweepHdr* __restrict__ hp,
                const AOp* __restrict__ ops, const double2* __restrict__ pool, double* partial) {
  adj_sweep_body(psi, lam, hp, ops, pool, partial, blockIdx.x, gridDim.x, blockIdx.x, ~0ULL,
                 gridDim.x);
}

// Sweep k of many independent (psi, lambda) pairs in one launch: job j is
// one parameter set's sweep, split into chunks of chunk_tiles consecutive
// tiles; the CTAs take (job, chunk) work items in order.  Chunk c of job j
// writes its sums to jobs[j].partial[slot * nchunks + c].
__global__ void __launch_bounds__(kAThreads, 2)
    k_adj_sweep_multi(const AJob* __restrict__ jobs, uint32_t njobs, uint32_t nchunks,
                      uint64_t chunk_tiles) {
  const uint64_t work = (uint64_t)njobs * nchunks;
  for (uint64_t w = blockIdx.x; w < work; w += gridDim.x) {
    const AJob J = jobs[w / nchunks];
    const uint32_t c = (uint32_t)(w % nchunks);
    adj_sweep_body(J.psi, J.lam, J.hdr, J.ops, J.pool, J.partial, c, nchunks, c * chunk_tiles,
                   (c + 1) * chunk_tiles, 1);
    __syncthreads();
  }
}

// jobs[j].out[map[s]] = sum over chunks (in order) of jobs[j].partial[s][chunk]
__global__ void k_adj_slots_multi(const AJob* __restrict__ jobs, uint32_t nchunks) {
  const AJob J = jobs[blockIdx.y];
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= J.nslots) return;
  double a = 0.0;
  for (uint32_t c = 0; c < nchunks; ++c) a += J.partial[(size_t)s * nchunks + c];
  J.out[J.map[s]] = a;
}

// out[map[s]] = sum over CTAs of partial[s][cta], a warp per slot (one thread
// per slot took 14 us a sweep for 296 CTAs)
__global__ void k_adj_slots(const double* partial, uint32_t nslots, uint32_t ctas,
                            const uint32_t* map, double* out) {
  const uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (s >= nslots) return;
  double a = 0.0;
  for (uint32_t c = lane; c < ctas; c += 32) a += partial[(size_t)s * ctas + c];
  a = warp_sum_d(a);
  if (lane == 0) out[map[s]] = a;
}

// ---- host planner ----------------------------------------------------------------------------

inline hc cjh(hc z) { return hc{z.re, -z.im}; }

// One gate of the reversed program, classified for the sweep.
struct AGate {
  int64_t inst;
  int kind;  // 0: one-qubit, 1: controlled one-qubit, 2: diagonal (<= 2 qubits), 3: dense 2q, 4: per-gate
  uint32_t t = 0, c = 0;      // target / control (kind 0, 1)
  uint32_t qa = 0, qb = 0;    // diagonal / dense qubits (qa = MSB)
  uint32_t nq = 0;            // diagonal: 1 or 2
  hc u[4];                    // kind 0/1: 2x2 (block)
  hc du[4][4];                // derivatives of the 2x2 (block)
  hc dg[4], ddg[4][4];        // kind 2: diagonal and its derivatives
  hc m4[16], dm4[16];         // kind 3: 4x4 and its derivative
  int np = 0;                 // active derivatives
  uint32_t slot0 = 0;         // first global slot
};

bool diag2(const hc u[4]) { return is_zero(u[1]) && is_zero(u[2]); }

}  // namespace

// Implemented in dq_adjoint.cu: 2x2 block + derivatives of a (controlled)
// one-qubit parametrised kind; derivatives of rxx / rzz.
bool adjoint_block_derivs(const dq_inst& in, hc u[4], hc d[4][4], int* np);
bool adjoint_rxx_rzz_deriv(const dq_inst& in, hc m[16], hc dm[16]);
bool adjoint_controlled_block(int kind);

namespace {

int classify_gate(const dq_inst& in, const int32_t* pidx, uint64_t r, uint32_t slot0, AGate& g) {
  g.inst = (int64_t)r;
  g.slot0 = slot0;
  int active[4] = {0, 0, 0, 0};
  int nact = 0;
  if (pidx)
    for (int j = 0; j < 4; ++j)
      if (pidx[4 * r + j] >= 0) active[nact++] = j;
  hc u[4], d[4][4];
  int np = 0;
  const bool param_block = adjoint_block_derivs(in, u, d, &np);
  if (param_block || matrix_1q(in.kind, in.p, u)) {
    const bool ctl = param_block ? adjoint_controlled_block(in.kind) : false;
    for (int i = 0; i < 4; ++i) g.u[i] = u[i];
    g.np = nact;
    for (int a = 0; a < nact; ++a)
      for (int i = 0; i < 4; ++i) g.du[a][i] = d[active[a]][i];
    // diagonal only if the matrix and every active derivative are (ry(0) is
    // the identity, its derivative is not diagonal) and at most one
    // parameter is active (u3(0, phi, lambda) with both angles trainable
    // stays a 2x2 op, which carries up to four derivatives)
    bool dg = diag2(u) && nact <= 1;
    for (int a = 0; a < nact; ++a) dg = dg && diag2(g.du[a]);
    if (!ctl) {
      g.t = (uint32_t)in.q[0];
      if (dg) {
        g.kind = 2;
        g.nq = 1;
        g.qa = g.t;
        g.dg[0] = u[0];
        g.dg[1] = u[3];
        for (int a = 0; a < nact; ++a) {
          g.ddg[a][0] = g.du[a][0];
          g.ddg[a][1] = g.du[a][3];
        }
      } else {
        g.kind = 0;
      }
      return DQ_OK;
    }
    g.c = (uint32_t)in.q[0];
    g.t = (uint32_t)in.q[1];
    if (dg) {  // controlled diagonal: a two-qubit diagonal (c = MSB)
      g.kind = 2;
      g.nq = 2;
      g.qa = g.c;
      g.qb = g.t;
      g.dg[0] = R(1); g.dg[1] = R(1); g.dg[2] = u[0]; g.dg[3] = u[3];
      for (int a = 0; a < nact; ++a) {
        g.ddg[a][0] = R(0); g.ddg[a][1] = R(0);
        g.ddg[a][2] = g.du[a][0]; g.ddg[a][3] = g.du[a][3];
      }
    } else {
      g.kind = 1;
    }
    return DQ_OK;
  }
  if (nact > 0 && !(in.kind == DQ_RXX || in.kind == DQ_RZZ))
    return fail(DQ_ERR_INTERNAL, "parameter slot on a kind without a derivative");
  Gate gt;
  if (!matrix_nq(in, gt)) return fail(DQ_ERR_INTERNAL, "instruction kind without a matrix");
  if (gt.k > 2) {
    g.kind = 4;
    return DQ_OK;
  }
  hc dm[16];
  for (int i = 0; i < 16; ++i) dm[i] = R(0);
  if (nact) adjoint_rxx_rzz_deriv(in, gt.m, dm);
  g.np = nact;
  GateOp op;
  classify(gt, op);
  g.qa = gt.qubits[0];
  g.qb = gt.qubits[1];
  if (nact == 0 && (op.cls == GC_ONE_Q || op.cls == GC_PHASE || op.cls == GC_XPERM)) {
    // controlled one-qubit without a trainable parameter (rxx / rzz at
    // special angles with an active slot keep their 4x4 and derivative)
    g.c = gt.qubits[0];
    g.t = gt.qubits[1];
    for (int i = 0; i < 4; ++i) g.u[i] = hc{0, 0};
    g.u[0] = gt.m[10]; g.u[1] = gt.m[11]; g.u[2] = gt.m[14]; g.u[3] = gt.m[15];
    if (diag2(g.u)) {
      g.kind = 2;
      g.nq = 2;
      g.qa = g.c;
      g.qb = g.t;
      g.dg[0] = R(1); g.dg[1] = R(1); g.dg[2] = g.u[0]; g.dg[3] = g.u[3];
    } else {
      g.kind = 1;
    }
    return DQ_OK;
  }
  bool dgn = true;
  for (int r2 = 0; r2 < 4; ++r2)
    for (int c2 = 0; c2 < 4; ++c2)
      if (r2 != c2 && (!is_zero(gt.m[r2 * 4 + c2]) || (nact && !is_zero(dm[r2 * 4 + c2]))))
        dgn = false;
  if (dgn) {
    g.kind = 2;
    g.nq = 2;
    for (int i = 0; i < 4; ++i) {
      g.dg[i] = gt.m[i * 5];
      if (nact) g.ddg[0][i] = dm[i * 5];
    }
    return DQ_OK;
  }
  g.kind = 3;
  for (int i = 0; i < 16; ++i) {
    g.m4[i] = gt.m[i];
    g.dm4[i] = dm[i];
  }
  return DQ_OK;
}

struct ASweepPlan {
  uint64_t Lmask = 0;
  std::vector<AGate> gates;  // reverse program order
};

// Qubits a gate needs local.
uint64_t need_local(const AGate& g) {
  switch (g.kind) {
    case 0: case 1: return 1ULL << g.t;
    case 3: return (1ULL << g.qa) | (1ULL << g.qb);
    default: return 0;
  }
}

void push_mats(std::vector<double2>& pool, const hc* m, int count) {
  for (int i = 0; i < count; ++i) pool.push_back(make_double2(m[i].re, m[i].im));
}

// D' = dU V (V = U^dagger, both 2x2 row-major): the derivative in the form
// that acts on the amplitudes before the op.  Parts below 1e-14 of the
// largest are rounding residue of exact zeros (ry: dU V = -i Y / 2) and are
// stored as zeros, which the register phases skip.
void push_dprime(std::vector<double2>& pool, const hc du[4], const hc v[4]) {
  hc d[4];
  double mx = 0.0;
  for (int r = 0; r < 2; ++r)
    for (int c = 0; c < 2; ++c) {
      const hc x = du[2 * r] * v[c] + du[2 * r + 1] * v[2 + c];
      d[2 * r + c] = x;
      mx = std::max(mx, std::max(std::fabs(x.re), std::fabs(x.im)));
    }
  for (hc& x : d) {
    if (std::fabs(x.re) <= 1e-14 * mx) x.re = 0.0;
    if (std::fabs(x.im) <= 1e-14 * mx) x.im = 0.0;
  }
  push_mats(pool, d, 4);
}

// A diagonal gate's angle polynomial and Walsh weights: its entries are
// V[2 b0 + b1] = exp(i (al + be b0 + ga b1 + de b0 b1)), and a gradient term is
// sum_S w[S] (Walsh coefficient of Im(conj(lambda) psi) on the bits in S).
// A one-qubit diagonal (entry index b0) is the same with b1 = 0: its weights
// with S1 = 1 vanish.
struct DiagPoly {
  double al, be, ga, de;
  double w[4];
  bool ok;  // dU U^dagger is imaginary (all supported kinds)
};
DiagPoly diag_poly(const AGate& g) {
  DiagPoly r{};
  double th[4];
  hc x[4];
  const uint32_t D = 1u << g.nq;
  for (uint32_t e = 0; e < 4; ++e) {
    const uint32_t src = D == 4 ? e : (e >> 1);
    const hc v = cjh(g.dg[src]), d = g.np ? g.ddg[0][src] : hc{0, 0};
    th[e] = std::atan2(v.im, v.re);
    x[e] = v * d;
  }
  r.al = th[0];
  r.be = th[2] - th[0];
  r.ga = th[1] - th[0];
  r.de = th[3] - th[2] - th[1] + th[0];
  double mx = 0.0, re = 0.0;
  for (int e = 0; e < 4; ++e) {
    mx = std::max(mx, std::fabs(x[e].im));
    re = std::max(re, std::fabs(x[e].re));
  }
  r.ok = !(re > 1e-13);
  for (int S = 0; S < 4; ++S) {
    double im = 0.0;
    for (int e = 0; e < 4; ++e) im += (((e >> 1) & (S >> 1)) ^ (e & S & 1)) ? -x[e].im : x[e].im;
    // parts below 1e-14 of the largest entry are rounding residue of zeros
    r.w[S] = std::fabs(0.25 * im) <= 1e-14 * mx ? 0.0 : -0.25 * im;
  }
  return r;
}

// Where a qubit's bit is during a pass: register bit (8 + k), bit of
// threadIdx.x (0..7), or bit of the tile's base (64 + qubit).
struct PassBits {
  uint32_t code[64];
};

// Appends the record of a run of diagonal gates; sigma: what both vectors
// carry at that point; pre: the factor the run applies.
void push_drun(std::vector<double2>& blob, const std::vector<AGate>& gates, const std::vector<uint32_t>& run,
               const std::vector<uint32_t>& slot, const PassBits& pb, long double sigma, long double pre,
               uint32_t tab) {
  const long double kTwoPi = 2.0L * 3.14159265358979323846264338327950288L;
  long double c0 = 0.0L, H[3] = {0.0L, 0.0L, 0.0L};
  std::map<uint32_t, long double> loc[4], cst, lin;
  auto single = [&](uint32_t c, double x) {
    if (c >= 64) cst[(c - 64) | 63u << 6] += x;
    else if (c >= 8) loc[c - 7][0] += x;
    else loc[0][1u << c] += x;
  };
  auto pair = [&](uint32_t c, uint32_t d, double x) {
    if (c > d) std::swap(c, d);
    if (c >= 64) cst[(c - 64) | (d - 64) << 6] += x;
    else if (d >= 64) lin[c | (d - 64) << 4] += x;
    else if (c >= 8) H[c + d - 17] += x;
    else if (d >= 8) loc[d - 7][1u << c] += x;
    else loc[0][1u << c | 1u << d] += x;
  };
  std::vector<DTerm> layer[4];
  const double wt = (double)(1.0L / (sigma * sigma));
  for (uint32_t i : run) {
    const AGate& g = gates[i];
    const DiagPoly p = diag_poly(g);
    const uint32_t ca = pb.code[g.qa], cb = g.nq == 2 ? pb.code[g.qb] : 0;
    c0 += p.al;
    if (p.be != 0.0) single(ca, p.be);
    if (g.nq == 2 && p.ga != 0.0) single(cb, p.ga);
    if (g.nq == 2 && p.de != 0.0) pair(ca, cb, p.de);
    if (!g.np) continue;
    uint32_t nt = 0;
    for (uint32_t S = 0; S < 4; ++S) {
      if (p.w[S] == 0.0) continue;
      uint32_t R = 0, T = 0, nb = 0, base[2] = {63u, 63u};
      for (uint32_t a = 0; a < 2; ++a) {
        if (!(S >> (1 - a) & 1u)) continue;
        const uint32_t c = a ? cb : ca;
        if (c >= 64) base[nb++] = c - 64;
        else if (c >= 8) R ^= 1u << (c - 8);
        else T ^= 1u << c;
      }
      DTerm d{};
      d.w = p.w[S] * wt;
      const uint32_t reg = (T >> 3 & 1u) | (T >> 4 & 1u) << 1 | (T >> 2 & 1u) << 2;
      d.code = (R | (T & 3u) << 3) | (T >> 5) << 5 | reg << 8 | base[0] << 11 | base[1] << 17;
      d.slot = slot[i];
      layer[nt++].push_back(d);
    }
  }
  // one term of a gate in a list (32 lanes take 32 terms and their slots at once)
  std::vector<DTerm> terms;
  uint32_t layers = 0;
  for (int k = 0; k < 4; ++k) {
    std::vector<DTerm>& l = layer[k];
    layers |= (uint32_t)l.size() << (8 * k);
    std::stable_sort(l.begin(), l.end(), [](const DTerm& x, const DTerm& y) { return (x.code >> 8 & 7u) < (y.code >> 8 & 7u); });
    for (size_t j = 0; j < l.size(); j += 32) {
      uint32_t used = 0;
      const size_t e = std::min(l.size(), j + 32);
      for (size_t x = j; x < e; ++x) used |= 1u << (l[x].code >> 8 & 7u);
      for (size_t x = j; x < e; ++x) l[x].code |= used << 23;
    }
    terms.insert(terms.end(), l.begin(), l.end());
  }
  auto put = [&](double x, double y) { blob.push_back(make_double2(x, y)); };
  auto put4 = [&](uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    const uint32_t v[4] = {a, b, c, d};
    double2 x;
    memcpy(&x, v, sizeof(x));
    blob.push_back(x);
  };
  auto angs = [&](const std::map<uint32_t, long double>& l) {
    for (auto& kv : l) {
      const DAng a{(double)remainderl(kv.second, kTwoPi), kv.first, 0};
      double2 x;
      memcpy(&x, &a, sizeof(x));
      blob.push_back(x);
    }
  };
  uint32_t ends = 0, n = 0, coupled = 0, pairs = 0;
  for (int k = 0; k < 4; ++k) {
    n += (uint32_t)loc[k].size();
    ends |= n << (8 * k);
  }
  for (auto& kv : lin) coupled |= 1u << (kv.first & 15u);
  for (int k = 0; k < 3; ++k)
    if (H[k] != 0.0L) pairs |= 1u << k;
  put((double)remainderl(c0, kTwoPi), (double)pre);
  for (int k = 0; k < 3; ++k) put((double)cosl(H[k]), (double)sinl(H[k]));
  put4((uint32_t)terms.size(), ends, (uint32_t)cst.size(), (uint32_t)lin.size());
  put4(coupled, pairs, tab, layers);
  for (const DTerm& d : terms) {
    double2 x;
    memcpy(&x, &d, sizeof(x));
    blob.push_back(x);
  }
  for (int k = 0; k < 4; ++k) angs(loc[k]);
  angs(cst);
  angs(lin);
}

// A rotation about Y or X (V = U^dagger, its derivative along the generator or
// none): its TanForm, tangent, scale and gradient weight.
bool tan_form(const AGate& g, uint32_t* form, double* t, long double* scale, double* kappa) {
  if (g.kind != 0 || g.np > 1) return false;
  const hc v[4] = {cjh(g.u[0]), cjh(g.u[2]), cjh(g.u[1]), cjh(g.u[3])};
  const bool y = v[0].im == 0.0 && v[1].im == 0.0 && v[2].im == 0.0 && v[3].im == 0.0 && v[0].re == v[3].re &&
                 v[1].re == -v[2].re;
  const bool x = !y && v[0].im == 0.0 && v[3].im == 0.0 && v[1].re == 0.0 && v[2].re == 0.0 &&
                 v[0].re == v[3].re && v[1].im == v[2].im;
  if (!y && !x) return false;
  *kappa = 0.0;
  if (g.np) {
    std::vector<double2> d;
    push_dprime(d, g.du[0], v);
    for (int e : {0, 3})
      if (d[e].x != 0.0 || d[e].y != 0.0) return false;
    const double lo = y ? d[1].x : d[1].y, hi = y ? -d[2].x : d[2].y;
    if ((y ? d[1].y : d[1].x) != 0.0 || (y ? d[2].y : d[2].x) != 0.0) return false;
    if (!(std::fabs(lo - hi) <= 1e-14 * std::fabs(hi))) return false;
    *kappa = y ? d[2].x : -d[2].y;
  }
  const long double c = v[0].re, s = y ? v[1].re : v[1].im;
  *t = (double)(s / c);
  const long double r = 1.0L / sqrtl(1.0L + (long double)*t * (long double)*t);
  *scale = c < 0.0L ? -r : r;
  *form = y ? TF_Y : TF_X;
  return r > 0x1p-20L;  // a rotation by almost pi is a general op (and a NaN one)
}

size_t asweep_smem(const ASweepHdr& h);

// Encodes one sweep's ops given its final local set.
int encode_asweep(const ASweepPlan& sp, uint32_t n, ASweepHdr& hdr, std::vector<AOp>& ops,
                  std::vector<double2>& pool, std::vector<uint32_t>& slot_map) {
  memset(&hdr, 0, sizeof(hdr));
  hdr.n = n;
  uint32_t lidx[64];
  uint32_t m = 0;
  for (uint32_t q = 0; q < n; ++q) {
    if (sp.Lmask >> q & 1ULL) {
      lidx[q] = m;
      hdr.lpos[m++] = q;
    } else {
      hdr.npos[hdr.npos_cnt++] = q;
    }
  }
  hdr.m = m;
  hdr.ntiles = 1ULL << (n - m);
  const std::vector<AGate>& gates = sp.gates;
  std::vector<uint32_t> slot(gates.size());
  uint32_t nslots = 0;
  for (size_t i = 0; i < gates.size(); ++i) {
    slot[i] = nslots;
    for (int a = 0; a < gates[i].np; ++a) slot_map.push_back(gates[i].slot0 + (uint32_t)a);
    nslots += (uint32_t)gates[i].np;
  }
  // Items: a pass (diagonal run and / or one-qubit group), or a single op
  struct Item {
    std::vector<uint32_t> diag, ones;
    int64_t single = -1;
    long double pre = 1.0L, post = 1.0L;
  };
  std::vector<Item> items;
  bool general = false;  // an op outside the passes has a derivative
  for (size_t i = 0; i < gates.size();) {
    if (m >= 3 && gates[i].kind == 2 && diag_poly(gates[i]).ok) {
      Item it;
      for (; i < gates.size() && gates[i].kind == 2 && diag_poly(gates[i]).ok; ++i) it.diag.push_back((uint32_t)i);
      if (it.diag.size() == 1) {
        // by itself: a run's transform and factors cost more than a pass of its own
        // (14 qubits, rx and rz on each qubit in turn, crx ring: 0.58 ms of sweeps with
        // runs of one gate, 0.53 without)
        it.single = it.diag[0];
        general = general || gates[it.diag[0]].np;
        it.diag.clear();
      }
      items.push_back(it);
      continue;
    }
    if (m >= 3 && gates[i].kind == 0) {
      std::vector<uint32_t> run;
      uint64_t seen = 0;
      bool distinct = true;
      for (; i < gates.size() && gates[i].kind == 0; ++i) {
        distinct = distinct && !(seen >> gates[i].t & 1ULL);
        seen |= 1ULL << gates[i].t;
        run.push_back((uint32_t)i);
      }
      // ops on distinct qubits commute: the low local bits first, so that the
      // last pass can write to memory in whole 128-byte runs
      if (distinct)
        std::sort(run.begin(), run.end(), [&](uint32_t x, uint32_t y) { return lidx[gates[x].t] < lidx[gates[y].t]; });
      for (size_t k = 0; k < run.size();) {
        std::vector<uint32_t> grp;
        uint64_t bits = 0;
        for (; k < run.size() && grp.size() < kAPhaseOps; ++k) {
          const uint64_t b = bits | 1ULL << gates[run[k]].t;
          if (__builtin_popcountll(b) > 3) break;
          bits = b;
          grp.push_back(run[k]);
        }
        if (items.empty() || items.back().single >= 0 || !items.back().ones.empty()) items.push_back(Item());
        items.back().ones = grp;
      }
      continue;
    }
    Item it;
    it.single = (int64_t)i;
    general = general || gates[i].np;
    items.push_back(it);
    ++i;
  }
  // A pass for one op has fewer threads at work than a pair of amplitudes a thread
  // (its scale is its own already where other ops have derivatives): 9 qubits, as
  // above, 0.19 ms, 0.26 with passes of one op; 11 qubits 0.33 and 0.37.
  if (general)
    for (Item& it : items)
      if (it.single < 0 && it.diag.empty() && it.ones.size() == 1) {
        it.single = it.ones[0];
        it.ones.clear();
      }
  // The rotations' scales: one factor for the sweep, applied by its first
  // diagonal run or else after its last rotation; with derivatives outside
  // the passes each pass applies its own.
  long double total = 1.0L;
  int first_diag = -1, last_tan = -1;
  std::vector<long double> own(items.size(), 1.0L);
  std::vector<uint8_t> tan(gates.size(), 0);
  for (size_t k = 0; k < items.size(); ++k) {
    if (!items[k].diag.empty() && first_diag < 0) first_diag = (int)k;
    for (uint32_t i : items[k].ones) {
      uint32_t f;
      double t, kp;
      long double c;
      if (!tan_form(gates[i], &f, &t, &c, &kp) || fabsl(total * c) < 0x1p-300L) continue;
      tan[i] = 1;
      own[k] *= c;
      total *= c;
      last_tan = (int)k;
    }
  }
  if (general) {
    for (size_t k = 0; k < items.size(); ++k) (items[k].diag.empty() ? items[k].post : items[k].pre) = own[k];
  } else if (last_tan >= 0) {
    if (first_diag >= 0) items[(size_t)first_diag].pre = total;
    else items[(size_t)last_tan].post = total;
  }
  for (const Item& it : items)
    if (!it.diag.empty()) ++hdr.ndrun;
  std::vector<double2> blob((hdr.ndrun + 3) / 4, make_double2(0.0, 0.0));
  std::vector<uint32_t> doff;
  long double sigma = 1.0L;  // both vectors' factor at this point
  uint32_t pops = 0, min_last = 0;
  bool last_pass = false;
  auto push_one = [&](uint32_t i) {
    const AGate& g = gates[i];
    AOp op{};
    op.np = (uint8_t)g.np;
    op.slot = slot[i];
    op.sel = -1;
    op.mat = (uint32_t)pool.size();
    op.type = A_ONE;
    op.lt = (uint8_t)lidx[g.t];
    const hc v[4] = {cjh(g.u[0]), cjh(g.u[2]), cjh(g.u[1]), cjh(g.u[3])};
    if (g.kind == 1 && !(sp.Lmask >> g.c & 1ULL)) {
      // non-local control: variant 0 (control 0) is the identity
      op.sel = (int8_t)g.c;
      op.skip0 = 1;
      const hc id[4] = {R(1), R(0), R(0), R(1)};
      push_mats(pool, id, 4);
      for (int a = 0; a < g.np; ++a) {
        const hc z[4] = {R(0), R(0), R(0), R(0)};
        push_mats(pool, z, 4);
      }
    } else if (g.kind == 1) {
      op.lctrl = 1u << lidx[g.c];
    }
    push_mats(pool, v, 4);
    for (int a = 0; a < g.np; ++a) push_mats(pool, g.du[a], 4);
    if (g.kind == 0)
      for (int a = 0; a < g.np; ++a) push_dprime(pool, g.du[a], v);
    ops.push_back(op);
  };
  for (const Item& it : items) {
    last_pass = false;
    if (it.single >= 0) {
      const uint32_t i = (uint32_t)it.single;
      const AGate& g = gates[i];
      if (g.kind == 0 || g.kind == 1) {
        push_one(i);
        continue;
      }
      AOp op{};
      op.np = (uint8_t)g.np;
      op.slot = slot[i];
      op.sel = -1;
      op.mat = (uint32_t)pool.size();
      if (g.kind == 3) {
        op.type = A_TWO;
        op.lt = (uint8_t)lidx[g.qa];
        op.lt2 = (uint8_t)lidx[g.qb];
        hc v[16];
        for (int r = 0; r < 4; ++r)
          for (int c = 0; c < 4; ++c) v[r * 4 + c] = cjh(g.m4[c * 4 + r]);
        push_mats(pool, v, 16);
        if (g.np) push_mats(pool, g.dm4, 16);
      } else {
        if (g.np > 1) return fail(DQ_ERR_INTERNAL, "diagonal op with more than one derivative");
        op.type = A_DIAG;
        op.ndq = (uint8_t)g.nq;
        const uint32_t qs[2] = {g.qa, g.qb};
        for (uint32_t a = 0; a < g.nq; ++a)
          op.dq[a] = (sp.Lmask >> qs[a] & 1ULL) ? (uint8_t)(0x80u | lidx[qs[a]]) : (uint8_t)qs[a];
        hc v[4] = {R(1), R(1), R(1), R(1)}, dd[4] = {R(0), R(0), R(0), R(0)};
        for (uint32_t e = 0; e < (1u << g.nq); ++e) {
          v[e] = cjh(g.dg[e]);
          if (g.np) dd[e] = g.ddg[0][e];
        }
        push_mats(pool, v, 4);
        if (g.np) push_mats(pool, dd, 4);
      }
      ops.push_back(op);
      continue;
    }
    AOp h{};
    h.type = A_PASS;
    h.cnt = (uint8_t)it.ones.size();
    h.mat = kNone;
    // register bits: the targets, then the highest other local bits
    std::vector<uint32_t> bits;
    auto add_bit = [&](uint32_t b) {
      if (std::find(bits.begin(), bits.end(), b) == bits.end()) bits.push_back(b);
    };
    for (uint32_t i : it.ones) add_bit(lidx[gates[i].t]);
    for (uint32_t b = m; b-- > 0 && bits.size() < 3;) add_bit(b);
    h.lt = (uint8_t)bits[0];
    h.lt2 = (uint8_t)bits[1];
    h.dq[0] = (uint8_t)bits[2];
    last_pass = true;
    min_last = *std::min_element(bits.begin(), bits.end());
    if (!it.diag.empty()) {
      PassBits pb;
      uint32_t rank = 0;
      for (uint32_t q = 0; q < n; ++q) {
        if (!(sp.Lmask >> q & 1ULL)) {
          pb.code[q] = 64 + q;
          continue;
        }
        const size_t k = (size_t)(std::find(bits.begin(), bits.end(), lidx[q]) - bits.begin());
        pb.code[q] = k < 3 ? 8u + (uint32_t)k : rank++;
      }
      h.ndq = 1;
      h.dq[1] = (uint8_t)doff.size();
      h.slot = (uint32_t)blob.size();
      for (uint32_t i : it.diag) h.np = (uint8_t)(h.np | (gates[i].np ? 1 : 0));
      doff.push_back((uint32_t)blob.size());
      push_drun(blob, gates, it.diag, slot, pb, sigma, it.pre, kNone);
      sigma *= it.pre;
    }
    // up to three rotations of one form on distinct qubits join the pass (the
    // register bits are their targets in order); other ops are a phase
    uint32_t form = 0;
    bool fast = it.ones.size() <= 3;
    for (size_t k = 0; k < it.ones.size(); ++k) {
      const AGate& g = gates[it.ones[k]];
      uint32_t f = 0;
      double t, kp;
      long double c;
      fast = fast && tan[it.ones[k]] && lidx[g.t] == bits[k] && tan_form(g, &f, &t, &c, &kp) && (k == 0 || f == form);
      form = f;
    }
    size_t hi = ops.size();
    if (fast) {
      if (!it.ones.empty()) h.pad[0] = (uint8_t)(1 + form + 2 * (it.ones.size() - 1));
      ops.push_back(h);
    } else {
      if (h.ndq) {
        AOp d = h;
        d.cnt = 0;
        ops.push_back(d);
        h.ndq = h.np = h.dq[1] = 0;
        h.slot = 0;
        ++hi;
      }
      h.type = A_PHASE;
      ops.push_back(h);
      last_pass = false;
    }
    for (uint32_t i : it.ones) {
      push_one(i);
      uint32_t f;
      double t, kp;
      long double c;
      if (tan[i] && tan_form(gates[i], &f, &t, &c, &kp)) {
        AOp& op = ops.back();
        op.cnt = (uint8_t)(1 + f);
        op.lctrl = (uint32_t)pool.size();
        pool.push_back(make_double2(t, (double)((long double)kp / (sigma * sigma))));
        sigma /= c;
      } else {  // the derivatives of a general op carry the weight (D', the last entries pushed)
        const double wt = (double)(1.0L / (sigma * sigma));
        for (size_t e = pool.size() - 4 * (size_t)gates[i].np; e < pool.size(); ++e)
          pool[e] = make_double2(wt * pool[e].x, wt * pool[e].y);
      }
    }
    if (it.post != 1.0L) {
      ops[hi].mat = (uint32_t)pool.size();
      pool.push_back(make_double2((double)it.post, 0.0));
      sigma *= it.post;
    }
    pops += (uint32_t)it.ones.size();
  }
  for (size_t k = 0; k < doff.size(); ++k) memcpy(reinterpret_cast<uint32_t*>(blob.data()) + k, &doff[k], 4);
  hdr.direct = last_pass && min_last >= kALoMin;
  // passes' op data staged once per CTA when it fits
  if (pops <= kAPhaseStage) {
    uint32_t b = 0;
    for (AOp& o : ops)
      if (o.type == A_PASS || o.type == A_PHASE) {
        o.lctrl = b;
        b += o.cnt;
      }
    hdr.phase_ops = pops;
  }
  hdr.nops = (uint32_t)ops.size();
  hdr.nslots = nslots;
  hdr.nblob = (uint32_t)blob.size();
  hdr.blob0 = (uint32_t)pool.size();
  if (hdr.nops > kAMaxSweepOps) return fail(DQ_ERR_INTERNAL, "too many ops in an adjoint sweep");
  for (uint32_t off : doff) {
    ++hdr.ntab;
    if (hdr.ntiles < kATabTiles || asweep_smem(hdr) > kATwoCtas) {
      --hdr.ntab;
      break;
    }
    reinterpret_cast<uint32_t*>(blob.data() + off + 5)[2] = hdr.ntab - 1;  // DMask::tab
  }
  pool.insert(pool.end(), blob.begin(), blob.end());
  return DQ_OK;
}

// Dynamic shared memory of a sweep: psi and lambda tiles, phase tables, the
// diagonal runs' records and factors, per-warp gradient slots, the op list and
// the staged op data (layout as in adj_sweep_body).  At most 160 KB: 64 of tiles,
// 22 of records (4 terms and 3 angles a gate, 192 gates), 37 of factors (96 runs),
// 12 of slots, 21 of ops; tables are added up to kATwoCtas only.
size_t asweep_smem(const ASweepHdr& h) {
  const size_t nops2 = ((size_t)h.nops + 1) / 2 * 2;
  return sizeof(double2) * (2 * (size_t)(1u << h.m) + (size_t)h.ntab * 4 * kAThreads + h.nblob +
                            2 * kDFactors * (size_t)h.ndrun) +
         sizeof(double) * (h.nslots ? h.nslots : 1) * kAWarps + sizeof(AOp) * nops2 +
         sizeof(PSub) * (h.phase_ops ? h.phase_ops : kAPhaseOps);
}

// CTAs of a launch: two per SM.  Also lets the sweep kernels use all of an
// SM's shared memory (sweeps of many different ops need more than half).
int sweep_ctas(int device) {
  static std::mutex mu;
  static int ctas[64];
  std::lock_guard<std::mutex> lk(mu);
  if (ctas[device & 63] == 0) {
    int sms = 148, most = 0;
    DQ_CUDA_TRY(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
    DQ_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    for (const void* k : {(const void*)k_adj_sweep, (const void*)k_adj_sweep_multi}) {
      cudaFuncAttributes fa{};
      DQ_CUDA_TRY(cudaFuncGetAttributes(&fa, k));
      DQ_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       most - (int)fa.sharedSizeBytes));
    }
    ctas[device & 63] = 2 * sms;
  }
  return ctas[device & 63];
}

// Segments of the backward pass in backward order: fused sweeps and the
// instructions undone one at a time (three or more qubits).
struct BackSeg {
  bool sweep;
  ASweepPlan plan;
  int64_t inst;
};

int plan_backward_segments(uint32_t n, const dq_inst* prog, uint64_t ninst, const int32_t* pidx,
                           uint64_t nslots, std::vector<BackSeg>& segs) {
  // global slot numbering: program order, parameter order within a gate
  std::vector<uint32_t> first_slot(ninst + 1, 0);
  for (uint64_t i = 0; i < ninst; ++i) {
    uint32_t c = 0;
    if (pidx)
      for (int j = 0; j < 4; ++j) c += pidx[4 * i + j] >= 0;
    first_slot[i + 1] = first_slot[i] + c;
  }
  if (first_slot[ninst] != nslots) return fail(DQ_ERR_INTERNAL, "slot count mismatch");
  const uint32_t m_max = std::min<uint32_t>(n, kAMaxLocal);
  const uint32_t lo = std::min<uint32_t>(n, kALoMin);
  const uint64_t lo_mask = (1ULL << lo) - 1;
  ASweepPlan cur;
  cur.Lmask = lo_mask;
  uint32_t cur_slots = 0;
  auto close = [&]() {
    if (!cur.gates.empty()) {
      // widen the local set to m_max with the lowest unused qubits (more
      // work per tile, fewer tiles; the set only needs to contain the gates')
      for (uint32_t q = 0; q < n && (uint32_t)__builtin_popcountll(cur.Lmask) < m_max; ++q)
        cur.Lmask |= 1ULL << q;
      segs.push_back(BackSeg{true, cur, -1});
    }
    cur = ASweepPlan();
    cur.Lmask = lo_mask;
    cur_slots = 0;
  };
  for (uint64_t r = ninst; r-- > 0;) {
    const dq_inst& in = prog[r];
    if (in.kind == DQ_ID || in.kind == DQ_U0 || in.kind == DQ_BARRIER || in.kind == DQ_CLASSICAL ||
        in.kind == DQ_G_NOOP)
      continue;
    AGate g;
    DQ_TRY(classify_gate(in, pidx, r, first_slot[r], g));
    if (g.kind == 4) {
      close();
      segs.push_back(BackSeg{false, ASweepPlan(), (int64_t)r});
      continue;
    }
    const uint64_t need = need_local(g);
    const uint64_t widened = cur.Lmask | need;
    if ((uint32_t)__builtin_popcountll(widened) > m_max || cur.gates.size() >= kAMaxOps ||
        cur_slots + (uint32_t)g.np > kAMaxSlots) {
      close();
    }
    cur.Lmask |= need;
    cur.gates.push_back(g);
    cur_slots += (uint32_t)g.np;
  }
  close();
  return DQ_OK;
}

}  // namespace

int adjoint_backward_fused(double2* psi, double2* lam, uint32_t n, const dq_inst* prog,
                           uint64_t ninst, const int32_t* pidx, uint64_t nslots, double* d_slots,
                           cudaStream_t st, int device, AdjSweepStats* stats) {
  using Seg = BackSeg;
  std::vector<Seg> segs;
  DQ_TRY(plan_backward_segments(n, prog, ninst, pidx, nslots, segs));
  const int ctas_max = sweep_ctas(device);
  if (ctas_max <= 0) return DQ_ERR_CUDA;
  // device buffers for all sweeps at once
  std::vector<ASweepHdr> hdrs;
  std::vector<AOp> ops;
  std::vector<double2> pool;
  std::vector<uint32_t> slot_map;
  struct SweepRef {
    size_t hdr, op0, slot0;
    uint32_t nslots;
    unsigned grid;
  };
  std::vector<SweepRef> refs;
  size_t max_partial = 1;
  for (const Seg& s : segs) {
    if (!s.sweep) continue;
    ASweepHdr hdr;
    const size_t op0 = ops.size(), sl0 = slot_map.size();
    std::vector<AOp> o;
    DQ_TRY(encode_asweep(s.plan, n, hdr, o, pool, slot_map));
    for (AOp& a : o) ops.push_back(a);
    const unsigned grid = (unsigned)std::min<uint64_t>(hdr.ntiles, (uint64_t)ctas_max);
    refs.push_back(SweepRef{hdrs.size(), op0, sl0, hdr.nslots, grid});
    max_partial = std::max(max_partial, (size_t)hdr.nslots * grid);
    hdrs.push_back(hdr);
  }
  if (pool.empty()) pool.push_back(make_double2(0, 0));
  if (slot_map.empty()) slot_map.push_back(0);
  if (ops.empty()) ops.push_back(AOp{});
  if (hdrs.empty()) hdrs.push_back(ASweepHdr{});
  ASweepHdr* d_hdr = nullptr;
  AOp* d_ops = nullptr;
  double2* d_pool = nullptr;
  uint32_t* d_map = nullptr;
  double* d_part = nullptr;
  int rc = DQ_OK;
  auto cu = [&](cudaError_t e, const char* what) {
    if (e != cudaSuccess && rc == DQ_OK) {
      cudaGetLastError();
      rc = fail(e == cudaErrorMemoryAllocation ? DQ_ERR_OOM : DQ_ERR_CUDA,
                std::string(what) + ": " + cudaGetErrorString(e));
    }
  };
  cu(pool_malloc_async((void**)&d_hdr, sizeof(ASweepHdr) * hdrs.size(), st), "cudaMallocAsync(hdr)");
  cu(pool_malloc_async((void**)&d_ops, sizeof(AOp) * ops.size(), st), "cudaMallocAsync(ops)");
  cu(pool_malloc_async((void**)&d_pool, sizeof(double2) * pool.size(), st), "cudaMallocAsync(pool)");
  cu(pool_malloc_async((void**)&d_map, sizeof(uint32_t) * slot_map.size(), st), "cudaMallocAsync(map)");
  cu(pool_malloc_async((void**)&d_part, sizeof(double) * max_partial, st), "cudaMallocAsync(partials)");
  if (rc == DQ_OK) {
    cu(cudaMemcpyAsync(d_hdr, hdrs.data(), sizeof(ASweepHdr) * hdrs.size(), cudaMemcpyHostToDevice, st), "copy");
    cu(cudaMemcpyAsync(d_ops, ops.data(), sizeof(AOp) * ops.size(), cudaMemcpyHostToDevice, st), "copy");
    cu(cudaMemcpyAsync(d_pool, pool.data(), sizeof(double2) * pool.size(), cudaMemcpyHostToDevice, st), "copy");
    cu(cudaMemcpyAsync(d_map, slot_map.data(), sizeof(uint32_t) * slot_map.size(), cudaMemcpyHostToDevice, st), "copy");
  }
  size_t si = 0;
  uint64_t sweeps = 0, pergate = 0;
  for (const Seg& s : segs) {
    if (rc != DQ_OK) break;
    if (!s.sweep) {
      GateOp op;
      const dq_inst& in = prog[s.inst];
      hc u4[4];
      (void)u4;
      Gate gt;
      if (!matrix_nq(in, gt)) {
        rc = fail(DQ_ERR_INTERNAL, "instruction kind without a matrix");
        break;
      }
      const uint32_t D = 1u << gt.k;
      std::vector<hc> t(gt.m, gt.m + D * D);
      for (uint32_t r = 0; r < D; ++r)
        for (uint32_t c = 0; c < D; ++c) gt.m[r * D + c] = cjh(t[c * D + r]);
      classify(gt, op);
      rc = launch_gate(psi, n, op, st, device, nullptr);
      if (rc == DQ_OK) rc = launch_gate(lam, n, op, st, device, nullptr);
      ++pergate;
      continue;
    }
    const SweepRef& ref = refs[si++];
    const ASweepHdr& hdr = hdrs[ref.hdr];
    const size_t smem = asweep_smem(hdr);
    k_adj_sweep<<<ref.grid, kAThreads, smem, st>>>(psi, lam, d_hdr + ref.hdr, d_ops + ref.op0, d_pool,
                                                    d_part);
    cu(cudaGetLastError(), "k_adj_sweep");
    if (ref.nslots && rc == DQ_OK) {
      k_adj_slots<<<(ref.nslots + 3) / 4, 128, 0, st>>>(d_part, ref.nslots, ref.grid,
                                                            d_map + ref.slot0, d_slots);
      cu(cudaGetLastError(), "k_adj_slots");
    }
    ++sweeps;
  }
  if (d_hdr) cudaFreeAsync(d_hdr, st);
  if (d_ops) cudaFreeAsync(d_ops, st);
  if (d_pool) cudaFreeAsync(d_pool, st);
  if (d_map) cudaFreeAsync(d_map, st);
  if (d_part) cudaFreeAsync(d_part, st);
  if (stats) {
    stats->sweeps = sweeps;
    stats->pergate = pergate;
  }
  return rc;
}

// ---- many parameter sets at once -------------------------------------------------------

int adjoint_backward_plan_set(uint32_t n, const dq_inst* prog, uint64_t ninst, const int32_t* pidx,
                              uint64_t nslots, ABatchSet* out) {
  std::vector<BackSeg> segs;
  DQ_TRY(plan_backward_segments(n, prog, ninst, pidx, nslots, segs));
  ABatchSet s;
  for (const BackSeg& g : segs) {
    if (!g.sweep)
      return fail(DQ_ERR_UNSUPPORTED, "a gate of three or more qubits: no batched backward sweep");
    ASweepHdr hdr;
    std::vector<AOp> o;
    const size_t op0 = s.ops.size() / sizeof(AOp), sl0 = s.map.size();
    DQ_TRY(encode_asweep(g.plan, n, hdr, o, s.pool, s.map));
    s.ops.insert(s.ops.end(), reinterpret_cast<const uint8_t*>(o.data()),
                 reinterpret_cast<const uint8_t*>(o.data() + o.size()));
    s.op0.push_back(op0);
    s.slot0.push_back(sl0);
    s.nslots.push_back(hdr.nslots);
    s.hdrs.insert(s.hdrs.end(), reinterpret_cast<const uint8_t*>(&hdr),
                  reinterpret_cast<const uint8_t*>(&hdr + 1));
  }
  if (s.pool.empty()) s.pool.push_back(make_double2(0, 0));
  *out = std::move(s);
  return DQ_OK;
}

int adjoint_backward_batch(double2* const* psi, double2* const* lam, const std::vector<ABatchSet>& sets,
                           double* const* d_slots, cudaStream_t st, int device, uint64_t* launches) {
  const size_t B = sets.size();
  if (!B) return DQ_OK;
  // every set's headers, ops, pools and slot maps in four device arrays
  std::vector<ASweepHdr> hdrs;
  std::vector<AOp> ops;
  std::vector<double2> pool;
  std::vector<uint32_t> map;
  std::vector<size_t> bh(B), bo(B), bp(B), bm(B);
  size_t kmax = 0;
  for (size_t b = 0; b < B; ++b) {
    const ABatchSet& s = sets[b];
    bh[b] = hdrs.size();
    bo[b] = ops.size();
    bp[b] = pool.size();
    bm[b] = map.size();
    for (size_t k = 0; k < s.sweeps(); ++k) {
      ASweepHdr x;
      memcpy(&x, s.hdrs.data() + k * sizeof(ASweepHdr), sizeof(x));
      hdrs.push_back(x);
    }
    const size_t nops = s.ops.size() / sizeof(AOp);
    ops.resize(bo[b] + nops);
    if (nops) memcpy(ops.data() + bo[b], s.ops.data(), nops * sizeof(AOp));
    pool.insert(pool.end(), s.pool.begin(), s.pool.end());
    map.insert(map.end(), s.map.begin(), s.map.end());
    kmax = std::max(kmax, s.sweeps());
  }
  if (hdrs.empty()) return DQ_OK;
  if (ops.empty()) ops.push_back(AOp{});
  if (map.empty()) map.push_back(0);
  const int ctas = sweep_ctas(device);
  if (ctas <= 0) return DQ_ERR_CUDA;
  const uint64_t ntiles = hdrs[0].ntiles;
  const uint64_t chunk_tiles = std::max<uint64_t>(1, std::min<uint64_t>(64, ntiles));
  const uint32_t nchunks = (uint32_t)((ntiles + chunk_tiles - 1) / chunk_tiles);
  // jobs of every sweep index (device pointers filled in once the arrays exist)
  std::vector<AJob> jobs;
  std::vector<size_t> job_hdr, job_ops, job_pool, job_map;
  std::vector<size_t> job0(kmax + 1, 0);
  std::vector<size_t> smem(kmax, 0);
  std::vector<uint32_t> maxsl(kmax, 0);
  size_t part_per_job = 1;
  for (const ASweepHdr& h : hdrs) part_per_job = std::max<size_t>(part_per_job, (size_t)h.nslots * nchunks);
  for (size_t k = 0; k < kmax; ++k) {
    job0[k] = jobs.size();
    for (size_t b = 0; b < B; ++b) {
      const ABatchSet& s = sets[b];
      if (k >= s.sweeps()) continue;
      const ASweepHdr& h = hdrs[bh[b] + k];
      if (h.ntiles != ntiles) return fail(DQ_ERR_INTERNAL, "batched sweeps of unequal tile counts");
      AJob j{};
      j.psi = psi[b];
      j.lam = lam[b];
      j.out = d_slots[b];
      j.nslots = s.nslots[k];
      jobs.push_back(j);
      job_hdr.push_back(bh[b] + k);
      job_ops.push_back(bo[b] + s.op0[k]);
      job_pool.push_back(bp[b]);
      job_map.push_back(bm[b] + s.slot0[k]);
      smem[k] = std::max(smem[k], asweep_smem(h));
      maxsl[k] = std::max(maxsl[k], h.nslots);
    }
  }
  job0[kmax] = jobs.size();
  size_t max_jobs = 1;
  for (size_t k = 0; k < kmax; ++k) max_jobs = std::max(max_jobs, job0[k + 1] - job0[k]);
  ASweepHdr* d_hdr = nullptr;
  AOp* d_ops = nullptr;
  double2* d_pool = nullptr;
  uint32_t* d_map = nullptr;
  double* d_part = nullptr;
  AJob* d_jobs = nullptr;
  int rc = DQ_OK;
  auto cu = [&](cudaError_t e, const char* what) {
    if (e != cudaSuccess && rc == DQ_OK) {
      cudaGetLastError();
      rc = fail(e == cudaErrorMemoryAllocation ? DQ_ERR_OOM : DQ_ERR_CUDA,
                std::string(what) + ": " + cudaGetErrorString(e));
    }
  };
  // the device arrays come from the engine's size-keyed buffer cache: an
  // optimiser loop repeats their sizes, so its steps pay no cudaMalloc/cudaFree
  std::vector<std::pair<void*, size_t>> owned;
  auto take = [&](void** p, size_t bytes) {
    if (rc != DQ_OK) return;
    bytes = std::max<size_t>(bytes, 16);
    const int r = cache_alloc(device, bytes, p);
    if (r != DQ_OK) {
      rc = r;
      *p = nullptr;
      return;
    }
    owned.push_back({*p, bytes});
  };
  take((void**)&d_hdr, sizeof(ASweepHdr) * hdrs.size());
  take((void**)&d_ops, sizeof(AOp) * ops.size());
  take((void**)&d_pool, sizeof(double2) * pool.size());
  take((void**)&d_map, sizeof(uint32_t) * map.size());
  take((void**)&d_part, sizeof(double) * part_per_job * max_jobs);
  take((void**)&d_jobs, sizeof(AJob) * std::max<size_t>(jobs.size(), 1));
  if (rc == DQ_OK) {
    for (size_t k = 0; k < kmax; ++k)
      for (size_t i = job0[k]; i < job0[k + 1]; ++i) {
        AJob& j = jobs[i];
        j.hdr = d_hdr + job_hdr[i];
        j.ops = d_ops + job_ops[i];
        j.pool = d_pool + job_pool[i];
        j.map = d_map + job_map[i];
        j.partial = d_part + (i - job0[k]) * part_per_job;
      }
    cu(cudaMemcpyAsync(d_hdr, hdrs.data(), sizeof(ASweepHdr) * hdrs.size(), cudaMemcpyHostToDevice, st), "copy");
    cu(cudaMemcpyAsync(d_ops, ops.data(), sizeof(AOp) * ops.size(), cudaMemcpyHostToDevice, st), "copy");
    cu(cudaMemcpyAsync(d_pool, pool.data(), sizeof(double2) * pool.size(), cudaMemcpyHostToDevice, st), "copy");
    cu(cudaMemcpyAsync(d_map, map.data(), sizeof(uint32_t) * map.size(), cudaMemcpyHostToDevice, st), "copy");
    cu(cudaMemcpyAsync(d_jobs, jobs.data(), sizeof(AJob) * jobs.size(), cudaMemcpyHostToDevice, st), "copy");
  }
  for (size_t k = 0; k < kmax && rc == DQ_OK; ++k) {
    const uint32_t nj = (uint32_t)(job0[k + 1] - job0[k]);
    if (!nj) continue;
    const uint64_t work = (uint64_t)nj * nchunks;
    const unsigned grid = (unsigned)std::min<uint64_t>(work, (uint64_t)ctas);
    k_adj_sweep_multi<<<grid, kAThreads, smem[k], st>>>(d_jobs + job0[k], nj, nchunks, chunk_tiles);
    cu(cudaGetLastError(), "k_adj_sweep_multi");
    if (launches) ++*launches;
    if (maxsl[k] && rc == DQ_OK) {
      k_adj_slots_multi<<<dim3((maxsl[k] + 127) / 128, nj), 128, 0, st>>>(d_jobs + job0[k], nchunks);
      cu(cudaGetLastError(), "k_adj_slots_multi");
      if (launches) ++*launches;
    }
  }
  cudaStreamSynchronize(st);
  for (auto& o : owned) cache_free(device, o.second, o.first);
  return rc;
}

}  // namespace dq
