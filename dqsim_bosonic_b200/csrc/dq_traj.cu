// dq_traj.cu — batched shot trajectories in one persistent launch.
//
// simulate_shots (statevector/simulator.rs:216-322) runs every shot as its
// own trajectory: a fresh |0..0> state, the fused program (types.rs:248-293,
// run_fused_par 870-884, run_instruction_par 638-864), mid-circuit measure /
// reset / conditionals, and ChaCha8Rng::seed_from_u64(base_seed + i).  Here
// each trajectory lives entirely in shared memory: a thread-block cluster of
// 2^cb CTAs holds one 2^n-amplitude state (2^(n-cb) amplitudes per CTA, at
// most 8192 = 128 KiB), so n <= 16 with clusters of up to 8 CTAs.  Gates on
// the low n-cb qubits touch one CTA's shared memory; gates on the top cb
// qubits pair elements across CTAs through distributed shared memory.  A
// measurement reduces p1 per CTA (fixed order), exchanges the cluster's
// partials, draws the outcome from the device ChaCha8 stream and collapses
// in place.
//
// Shots share work.  Two shots of one program that have drawn the same
// outcomes so far hold the same state bit for bit, so a cluster carries a
// state together with the list of the shots that are in it.  A measurement
// compares every listed shot's own draw with the state's p1; when both
// outcomes occur the state is saved (HBM) with one half of the list as a task
// for any idle cluster and the cluster goes on with the other half.  Each
// distinct outcome history is computed once instead of once per shot: the
// bound is the latency of one trajectory while histories are few, and the
// shared memory and FP64 throughput of one trajectory per shot once every
// shot is on its own.  4096 shots of 16 qubits with four measure / reset
// pairs: 205 ms with one trajectory per shot, 0.80 ms here (16 histories); with
// 16 random outcomes per shot, every shot soon on its own: 132 ms and 96 ms.
// Clusters take tasks until none is left or running; states otherwise stay in
// shared memory, and only classical registers are written out.
//
// Arithmetic is the exact per-gate arithmetic of dq_engine.cu (num-complex
// order, no FMA, zero matrix entries skipped), so amplitudes match the
// oracle's sequential shot bit for bit; p1 is summed in a different order,
// which can only change an outcome when the draw lies within rounding of
// p1 — such draws (|r - p1| < 1e-12) are counted and reported.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <chrono>
#include <string>
#include <thread>
#include <vector>

#include "dq_common.cuh"
#include "dq_fused.cuh"
#include "dq_gates.hpp"
#include "dq_handle.cuh"
#include "dq_rng.cuh"
#include "dq_sweep.cuh"

namespace cg = cooperative_groups;

namespace dq {
namespace {

constexpr uint32_t kLocalBitsMax = 13;  // 8192 amplitudes = 128 KiB per CTA
// Tile bits of the fused sweeps that HBM-resident batch items run (2^12
// amplitudes: 8 thread bits of the 256-thread CTA and 4 register bits).
constexpr int kHbmTileBits = 12;
constexpr uint32_t kTrajMaxQubits = 16;
constexpr uint32_t kTrajMaxCbits = 1024;

enum TOpType : uint8_t {
  T_NOP = 0, T_ONEQ, T_PHASE, T_XPERM, T_SWAP, T_DIAG, T_DENSE, T_MEASURE, T_RESET, T_FAIL,
  T_RPHASE  // header of k (>= 2) T_ONEQ / T_XPERM ops on the four local bits q[0..3]
};

struct TOp {
  uint8_t type;
  uint8_t k;        // DIAG / DENSE: qubit count
  uint8_t t1, t2;   // target(s)
  uint32_t cond_first, cond_count;
  int32_t cbit;     // MEASURE: classical bit; FAIL: unused
  uint32_t mat;     // offset into the matrix pool (double2 units)
  uint32_t remote;  // bit 0: touches cluster qubits or needs a cluster reduction; kOpMulti
  uint64_t ctrl;    // control mask (all must be 1)
  uint8_t q[8];     // DIAG / DENSE qubits, q[0] = MSB of the matrix index; RPHASE: register bits
  int64_t inst;     // original instruction index (-1: a fused 2x2)
};
static_assert(sizeof(TOp) == 48, "TOp layout");
constexpr uint32_t kOpMulti = 2u;  // TOp::remote: a gate on two or more qubits (call counts)

struct TProg {         // one program of a launch
  uint32_t ops_off, nops;
  uint32_t n, lb;       // qubits; amplitudes per CTA = 2^lb
  uint32_t ncbits, pad;
  uint64_t base_seed;   // shot s draws from seed_from_u64(base_seed + s) (wrapping)
  uint64_t cbits_off;   // shot s writes cbits_out[cbits_off + s * ncbits ...]
  double2* state_out;   // device: final state of shot s at + s * 2^n, or null
  // Items too large for a cluster's shared memory (batch items of 17+ qubits)
  // keep their state in HBM at `hbm` and run as fused tile sweeps: sweeps
  // [sweep_first, sweep_first + nsweeps) of the launch's sweep table, the
  // first one generating its tiles from the basis index `synth`.
  double2* hbm;
  uint32_t sweep_first, nsweeps;
  long long synth;
  // A run on a state handle (small_run): the state it starts from (null: the
  // basis state `basis`), the classical bits it starts with (null: unwritten)
  // and its gate and measurement counts (one-qubit, wider, measurements)
  const double2* state_in;
  const int32_t* cbits_in;
  unsigned long long* counts;
  uint64_t basis;
};
struct TSweep {          // one fused sweep of an HBM item
  uint64_t off;          // byte offset of its program in the launch's sweep blob
  uint32_t ntiles, run_bits;
  uint32_t prog_bytes, micro;  // micro: the program has rotation phases
};
struct TItem {          // shots [shot, shot + count) of a program
  uint32_t prog, count;
  uint64_t shot;
};
// A state saved at a measurement, to be collapsed to `outcome` and run on for
// the shots order[src][lo .. hi).  Without a slot (more states than slots) the
// program is run from the start instead: the listed shots draw the same
// outcomes again.
struct alignas(16) TTask {
  uint32_t prog, oi;      // op index of the measurement
  uint32_t lo, hi, src;
  int32_t slot;
  uint32_t outcome, draws;
  double p1;
};
static_assert(sizeof(TTask) == 48, "TTask is read as three 16-byte words");
struct TrajParams {
  const TOp* ops;
  const double2* pool;
  const dq_cond* conds;
  const TProg* progs;
  const TItem* items;
  int32_t* cbits_out;
  unsigned long long* queue;     // [0] next item or task, [1] tasks pushed, [2] items and tasks unfinished
  unsigned long long* boundary;  // draws within 1e-12 of p1
  long long* failed;             // lowest (prog << 40 | instruction) that failed
  // shared shots (nslots and tasks are 0 / null when every item is one shot)
  uint32_t* order[2];            // shot lists, split from one into the other
  TTask* tasks;                  // at most one per shot
  int* ready;                    // task t is complete in memory
  double2* slots;                // nslots states of 2^n amplitudes
  int32_t* slot_cbits;           // nslots x ncbits
  const double* draws;           // draw k of shot s at s * draw_stride + k, or null
  uint32_t nslots, draw_stride;
  // ops, pool and conds as one image of stage_bytes at ops, copied to dynamic
  // shared memory at stage_at when the launch starts (0: read from memory; a
  // small program's op after op is otherwise a chain of L2 round trips)
  uint32_t stage_bytes, stage_at;
  uint64_t nitems;
  const uint8_t* sweep_blob;     // sweep programs of the HBM items (dq_sweep.cuh layout)
  const TSweep* sweeps;
};

__device__ __forceinline__ uint32_t ins0(uint32_t k, uint32_t p) {
  return ((k >> p) << (p + 1)) | (k & ((1u << p) - 1u));
}

// Shared-memory layout of a trajectory slice: logical element o lives at
// tswz(o).  The low three index bits are XORed with a fold of the higher ones
// so that eight threads touching elements that differ only in higher bits
// (pairs of a low target, strided controls) use eight different bank rows.
// The same bijection in every CTA keeps distributed-shared-memory accesses
// consistent; summation orders follow logical indices, so results are
// unchanged.
__device__ __forceinline__ uint32_t tswz(uint32_t o) {
  return o ^ (((o >> 3) ^ (o >> 6) ^ (o >> 9) ^ (o >> 12)) & 7u);
}

// One op of a register phase on the 16 amplitudes a thread holds (register
// index bit b = local qubit q[b] of the phase): the exact per-pair arithmetic
// of the shared-memory path, for the pairs whose control bits (creg) are set.
template <int RT>
__device__ __forceinline__ void rphase_1q(double2 (&a)[16], const double2 (&u)[4], uint32_t creg) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    if (j & (1 << RT)) continue;
    if (((uint32_t)j & creg) != creg) continue;
    const int k = j | (1 << RT);
    const double2 x = a[j], y = a[k];
    a[j] = cadd_x(cmul_x(u[0], x), cmul_x(u[1], y));
    a[k] = cadd_x(cmul_x(u[2], x), cmul_x(u[3], y));
  }
}
template <int RT>
__device__ __forceinline__ void rphase_x(double2 (&a)[16], uint32_t creg) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    if (j & (1 << RT)) continue;
    if (((uint32_t)j & creg) != creg) continue;
    const int k = j | (1 << RT);
    const double2 x = a[j];
    a[j] = a[k];
    a[k] = x;
  }
}

// Fixed-order block sum, result broadcast to every thread.
template <int THREADS>
__device__ double block_sum_all(double v, double* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_down_sync(0xffffffffu, v, o));
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0;
    for (int i = 0; i < THREADS / 32; ++i) a = __dadd_rn(a, sh[i]);
    sh[32] = a;
  }
  __syncthreads();
  return sh[32];
}

// The first draws of every shot, one thread per ChaCha8 block of eight.
__global__ void __launch_bounds__(128) k_traj_draws(const TProg* prog, uint64_t shots, uint32_t blocks,
                                                    double* out) {
  const uint64_t i = (uint64_t)blockIdx.x * 128 + threadIdx.x;
  if (i >= shots * blocks) return;
  uint32_t key[8], w[16];
  seed_key_from_u64(prog->base_seed + i / blocks, key);
  chacha8_stream_block(key, i % blocks, w);
#pragma unroll
  for (int k = 0; k < 8; ++k)
    out[i * 8 + k] = u64_to_f64((uint64_t)w[2 * k] | ((uint64_t)w[2 * k + 1] << 32));
}

__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// The next item (index below nitems) or task (nitems + t) to run; ~0 when
// nothing is left.  A cluster that finds none while others still run waits for
// what they may push, with a limit (seconds): leaving early is safe,
// the clusters that push also take tasks.
__device__ unsigned long long next_work(const TrajParams& P) {
  for (int tries = 0; tries < (1 << 21); ++tries) {
    unsigned long long h, t;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(h), "=l"(t) : "l"(P.queue) : "memory");
    if (h < P.nitems || (t > h - P.nitems && ld_acquire(P.ready + (h - P.nitems)))) {
      if (atomicCAS(P.queue, h, h + 1) == h) return h;
      continue;
    }
    if (!P.tasks || ld_acquire(P.queue + 2) == 0) break;
    __nanosleep(100);
  }
  return ~0ULL;
}

template <int THREADS>
__global__ void __launch_bounds__(THREADS) k_traj(const TrajParams P) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ double s_bcast[2];
  __shared__ int s_skip[2];  // double-buffered by op parity: one barrier per op suffices
  __shared__ unsigned long long s_item;
  __shared__ uint32_t s_count[2];   // a split's shots with outcome 0 and 1
  __shared__ unsigned long long s_task;

  cg::cluster_group cl = cg::this_cluster();
  const uint32_t C = cl.num_blocks(), rank = cl.block_rank();
  const uint32_t tid = threadIdx.x;
  const TOp* ops = P.ops;
  const double2* pool = P.pool;
  const dq_cond* conds = P.conds;
  if (P.stage_bytes) {
    uint8_t* st = smraw + P.stage_at;
    for (uint32_t i = tid * 16u; i < P.stage_bytes; i += THREADS * 16u)
      *reinterpret_cast<uint4*>(st + i) = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const uint8_t*>(P.ops) + i));
    ops = reinterpret_cast<const TOp*>(st);
    pool = reinterpret_cast<const double2*>(st + (reinterpret_cast<const uint8_t*>(P.pool) - reinterpret_cast<const uint8_t*>(P.ops)));
    conds = reinterpret_cast<const dq_cond*>(st + (reinterpret_cast<const uint8_t*>(P.conds) - reinterpret_cast<const uint8_t*>(P.ops)));
    __syncthreads();
  }
  auto sync_all = [&](bool cluster) {
    if (cluster && C > 1) cl.sync(); else __syncthreads();
  };

  for (;;) {
    // rank 0 takes the next item or task from the queue and shares it
    if (rank == 0 && tid == 0) s_item = next_work(P);
    sync_all(true);
    const unsigned long long item = (rank == 0) ? s_item : *cl.map_shared_rank(&s_item, 0);
    if (item == ~0ULL) {
      sync_all(true);  // no CTA leaves while another still reads its shared memory
      break;
    }
    TItem it;
    TTask tk{};
    uint32_t lo = 0, hi = 1, src = 2;  // the shots: order[src][lo .. hi), src 2: it.shot + lo .. hi
    if (item < P.nitems) {
      it = P.items[item];
      hi = it.count;
      tk.slot = -1;
    } else {
      const uint4* rec = reinterpret_cast<const uint4*>(P.tasks + (item - P.nitems));
      uint4 w[3];
      for (int i = 0; i < 3; ++i) w[i] = __ldcg(rec + i);
      memcpy(&tk, w, sizeof(tk));
      it.prog = tk.prog;
      it.shot = 0;
      lo = tk.lo;
      hi = tk.hi;
      src = tk.src;
    }
    auto shot_at = [&](uint32_t i) -> uint64_t {
      return src == 2 ? it.shot + i : (uint64_t)__ldcg(P.order[src] + i);
    };
    const TProg pg = P.progs[it.prog];
    if (pg.hbm) {
      // HBM item: the cluster's CTAs split the tiles of each sweep (tiles
      // rank, rank + C, ...; 256 threads run the 8-thread-bit geometry the
      // sweeps were planned for) with a cluster barrier between sweeps; the
      // fence makes each sweep's stores visible to the CTAs of the next one.
      // Each sweep's program is staged in shared memory behind two tile
      // buffers (the next tile loads while the current one is computed).
      if constexpr (THREADS == 256) {
        double2* bufs = reinterpret_cast<double2*>(smraw);
        double2* slots = bufs + 2 * (1u << kHbmTileBits);
        uint8_t* sprog = reinterpret_cast<uint8_t*>(slots + kMaxSlots);
        if (pg.nsweeps == 0) {  // nothing but a basis state to write
          const uint64_t len = 1ULL << pg.n;
          for (uint64_t i = (uint64_t)rank * THREADS + tid; i < len; i += (uint64_t)C * THREADS)
            pg.hbm[i] = make_double2(i == (uint64_t)pg.synth ? 1.0 : 0.0, 0.0);
        }
        for (uint32_t s = 0; s < pg.nsweeps; ++s) {
          const TSweep sw = P.sweeps[pg.sweep_first + s];
          const long long sy = s == 0 ? pg.synth : -1LL;
          for (uint32_t i = tid * 16u; i < sw.prog_bytes; i += THREADS * 16u)
            *reinterpret_cast<uint4*>(sprog + i) =
                __ldg(reinterpret_cast<const uint4*>(P.sweep_blob + sw.off + i));
          __syncthreads();
          if (sw.micro && sw.run_bits == 3)
            sweep_tiles<8, kHbmTileBits - 8, 2, 3, FORM_M>(pg.hbm, sprog, sw.ntiles, sy, bufs, slots, rank, C);
          else if (sw.micro)
            sweep_tiles<8, kHbmTileBits - 8, 2, 5, FORM_M>(pg.hbm, sprog, sw.ntiles, sy, bufs, slots, rank, C);
          else if (sw.run_bits == 3)
            sweep_tiles<8, kHbmTileBits - 8, 2, 3>(pg.hbm, sprog, sw.ntiles, sy, bufs, slots, rank, C);
          else
            sweep_tiles<8, kHbmTileBits - 8, 2, 5>(pg.hbm, sprog, sw.ntiles, sy, bufs, slots, rank, C);
          __threadfence();
          cl.sync();
        }
      }
      if (rank == 0)  // unitary items write no classical bit
        for (uint32_t i = tid; i < pg.ncbits; i += THREADS)
          P.cbits_out[pg.cbits_off + it.shot * pg.ncbits + i] = -1;
      sync_all(true);
      if (rank == 0 && tid == 0) atomicAdd(P.queue + 2, ~0ULL);
      continue;
    }
    const uint32_t lb = pg.lb, L = 1u << lb;
    double2* sm = reinterpret_cast<double2*>(smraw);
    double* red = reinterpret_cast<double*>(sm + L);    // [0..32]: block sums, [40]: CTA partial
    int32_t* cb = reinterpret_cast<int32_t*>(red + 48);  // classical bits
    const uint64_t gbase = (uint64_t)rank << lb;
    const uint64_t lmask = (uint64_t)L - 1;
    auto elem = [&](uint64_t g) -> double2* {
      const uint32_t r = (uint32_t)(g >> lb);
      double2* base = (r == rank) ? sm : cl.map_shared_rank(sm, r);
      return base + tswz((uint32_t)(g & lmask));
    };

    uint64_t draws = tk.draws;
    if (tk.slot >= 0) {  // slices are saved in their shared-memory layout
      const double2* s = P.slots + ((uint64_t)tk.slot << pg.n) + gbase;
#pragma unroll 4
      for (uint32_t i = tid; i < L; i += THREADS) sm[i] = __ldcg(s + i);
      for (uint32_t i = tid; i < pg.ncbits; i += THREADS)
        cb[i] = __ldcg(P.slot_cbits + (uint64_t)tk.slot * pg.ncbits + i);
    } else {
      draws = 0;
      for (uint32_t i = tid; i < L; i += THREADS)
        sm[tswz(i)] = pg.state_in ? pg.state_in[gbase + i] : make_double2(gbase + i == pg.basis ? 1.0 : 0.0, 0.0);
      for (uint32_t i = tid; i < pg.ncbits; i += THREADS) cb[i] = pg.cbits_in ? pg.cbits_in[i] : -1;
    }
    unsigned long long n1q = 0, nnq = 0, nmeas = 0;  // thread 0: executed gates and measurements
    bool last_cluster = true;
    sync_all(true);

    // divisor of a collapse (engine.rs:216-235)
    auto norm_of = [](int o, double p1) {
      const double q = o == 1 ? p1 : (1.0 - p1 < 0.0 ? 0.0 : 1.0 - p1);
      const double r = sqrt(q);
      return r < 1e-15 ? 1e-15 : r;
    };
    auto collapse = [&](const TOp& op, int o, double norm) {
      const uint32_t q = op.t1;
      const uint64_t qb = 1ULL << q;
      const double y = divisor(norm);
      for (uint32_t i = tid; i < L; i += THREADS) {
        const bool set = ((gbase | i) & qb) != 0;
        if (set != (o == 1)) {
          sm[tswz(i)] = make_double2(0.0, 0.0);
        } else {
          const double2 a = sm[tswz(i)];
          sm[tswz(i)] = make_double2(div_by(a.x, norm, y), div_by(a.y, norm, y));
        }
      }
      if (op.type == T_RESET && o == 1) {
        // X on q: an exact exchange of the two halves
        if (C > 1) cl.sync(); else __syncthreads();
        if (q < lb) {
          for (uint32_t k = tid; k < L / 2; k += THREADS) {
            const uint32_t a0 = ins0(k, q), a1 = a0 | (uint32_t)qb;
            const double2 x = sm[tswz(a0)];
            sm[tswz(a0)] = sm[tswz(a1)];
            sm[tswz(a1)] = x;
          }
        } else {
          const uint32_t tbr = 1u << (q - lb);
          if (!(rank & tbr)) {
            double2* other = cl.map_shared_rank(sm, rank | tbr);
            for (uint32_t i = tid; i < L; i += THREADS) {
              const double2 x = sm[i];
              sm[i] = other[i];
              other[i] = x;
            }
          }
        }
      }
    };
    uint32_t oi0 = 0;
    if (tk.slot >= 0) {  // finish the measurement the state was saved at
      const TOp op = ops[pg.ops_off + tk.oi];
      collapse(op, (int)tk.outcome, norm_of((int)tk.outcome, tk.p1));
      if (tid == 0 && op.type == T_MEASURE) cb[op.cbit] = (int)tk.outcome;
      oi0 = tk.oi + 1;
      sync_all(true);
    }

    // the next op's descriptor and one-qubit matrix are loaded while the
    // current op runs (global loads, otherwise a round trip before every op)
    TOp nxt{};
    double2 nu[4] = {};
    auto fetch = [&](uint32_t k) {
      nxt = ops[pg.ops_off + k];
      if (nxt.type == T_ONEQ)
        for (int i = 0; i < 4; ++i) nu[i] = pool[nxt.mat + i];
    };
    if (oi0 < pg.nops) fetch(oi0);
    for (uint32_t oi = oi0; oi < pg.nops; ++oi) {
      const TOp op = nxt;
      double2 u[4];
      for (int i = 0; i < 4; ++i) u[i] = nu[i];
      if (oi + 1 < pg.nops) fetch(oi + 1);
      // conditions (little-endian register value, unwritten bits read as 0)
      if (op.cond_count) {
        if (tid == 0) {
          int ok = 1;
          for (uint32_t c = 0; c < op.cond_count && ok; ++c) {
            const dq_cond cd = conds[op.cond_first + c];
            uint64_t actual = 0;
            for (uint64_t b = 0; b < cd.creg_size; ++b) {
              const uint64_t idx = cd.creg_base + b;
              const int32_t v = (idx < pg.ncbits) ? cb[idx] : 0;
              actual |= (uint64_t)(v > 0 ? v : 0) << b;
            }
            if (actual != cd.creg_value) ok = 0;
          }
          s_skip[oi & 1] = !ok;
        }
        __syncthreads();
        if (s_skip[oi & 1]) continue;
      }
      const bool remote = (op.remote & 1u) && C > 1;
      if (op.type == T_MEASURE || op.type == T_RESET) ++nmeas;
      else if (op.type != T_RPHASE && op.type != T_FAIL) (op.remote & kOpMulti ? nnq : n1q) += 1;
      if (remote && !last_cluster) cl.sync();

      switch (op.type) {
        case T_ONEQ:
        case T_XPERM: {
          const uint32_t t = op.t1;
          const uint64_t hi_ctrl = op.ctrl & ~lmask;
          const uint32_t lo_ctrl = (uint32_t)(op.ctrl & lmask);
          // local zero-insertion positions: target (if local) and local controls
          // local zero-insertion positions (the set bits of zmask, ascending;
          // no array: a dynamically indexed one would live in local memory)
          const uint64_t zmask = lo_ctrl | (t < lb ? (1ULL << t) : 0ULL);
          const int np = __popcll((long long)zmask);
          const uint32_t count = L >> np;
          const uint32_t p0 = np > 0 ? (uint32_t)(__ffsll((long long)zmask) - 1) : 0u;
          const uint64_t zm1 = zmask & (zmask - 1);
          const uint32_t p1 = np > 1 ? (uint32_t)(__ffsll((long long)zm1) - 1) : 0u;
          // pair k -> swizzled index of its element with the target bit 0
          auto index = [&](uint32_t k) -> uint32_t {
            uint32_t o;
            if (np == 1) {
              o = ins0(k, p0);
            } else if (np == 2) {
              o = ins0(ins0(k, p0), p1);
            } else {
              o = k;
              for (uint64_t mm = zmask; mm; mm &= mm - 1) o = ins0(o, (uint32_t)(__ffsll((long long)mm) - 1));
            }
            return tswz(o | lo_ctrl);
          };
          double2 *A, *B;
          uint32_t sx, lo, hi;
          if (t < lb) {
            if ((gbase & hi_ctrl) != hi_ctrl) break;
            A = B = sm;
            sx = tswz(1u << t);  // tswz is linear over XOR: partner = index ^ tswz(target bit)
            lo = 0;
            hi = count;
          } else {
            const uint32_t tbr = 1u << (t - lb);
            const uint32_t r0 = rank & ~tbr, r1 = rank | tbr;
            if ((((uint64_t)r0 << lb) & hi_ctrl) != hi_ctrl) break;
            A = (r0 == rank) ? sm : cl.map_shared_rank(sm, r0);
            B = (r1 == rank) ? sm : cl.map_shared_rank(sm, r1);
            sx = 0;
            const uint32_t half = count > 1 ? count >> 1 : 1;
            if (rank == r0) { lo = 0; hi = half; } else { lo = half; hi = count > 1 ? count : half; }
          }
          // four pairs per thread in flight: loads first, then the exact
          // per-pair arithmetic (pairs are disjoint, so the order of the
          // stores does not matter)
          for (uint32_t k0 = lo + tid; k0 < hi; k0 += 4u * THREADS) {
            uint32_t so[4];
            double2 a[4], b[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              const uint32_t k = k0 + (uint32_t)v * THREADS;
              so[v] = index(k < hi ? k : k0);
              a[v] = A[so[v]];
              b[v] = B[so[v] ^ sx];
            }
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              if (k0 + (uint32_t)v * THREADS >= hi) break;
              if (op.type == T_ONEQ) {
                A[so[v]] = cadd_x(cmul_x(u[0], a[v]), cmul_x(u[1], b[v]));
                B[so[v] ^ sx] = cadd_x(cmul_x(u[2], a[v]), cmul_x(u[3], b[v]));
              } else {
                A[so[v]] = b[v];
                B[so[v] ^ sx] = a[v];
              }
            }
          }
          break;
        }
        case T_PHASE: {
          const uint64_t need = op.ctrl | (1ULL << op.t1);
          const uint64_t hi = need & ~lmask, lo = need & lmask;
          if ((gbase & hi) != hi) break;
          const double2 e = pool[op.mat];
          const int np = __popcll((long long)lo);
          const uint32_t count = L >> np;
          const uint32_t p0 = np > 0 ? (uint32_t)(__ffsll((long long)lo) - 1) : 0u;
          const uint64_t lo1 = lo & (lo - 1);
          const uint32_t p1 = np > 1 ? (uint32_t)(__ffsll((long long)lo1) - 1) : 0u;
          for (uint32_t k0 = tid; k0 < count; k0 += 4u * THREADS) {
            uint32_t so[4];
            double2 a[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              const uint32_t k = k0 + (uint32_t)v * THREADS < count ? k0 + (uint32_t)v * THREADS : k0;
              uint32_t o;
              if (np == 1) {
                o = ins0(k, p0);
              } else if (np == 2) {
                o = ins0(ins0(k, p0), p1);
              } else {
                o = k;
                for (uint64_t mm = lo; mm; mm &= mm - 1) o = ins0(o, (uint32_t)(__ffsll((long long)mm) - 1));
              }
              so[v] = tswz(o | (uint32_t)lo);
              a[v] = sm[so[v]];
            }
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              if (k0 + (uint32_t)v * THREADS >= count) break;
              sm[so[v]] = cmul_x(e, a[v]);
            }
          }
          break;
        }
        case T_DIAG: {
          const uint32_t kq = op.k;
          for (uint32_t o = tid; o < L; o += THREADS) {
            const uint64_t g = gbase | o;
            uint32_t idx = 0;
            for (uint32_t b = 0; b < kq; ++b) idx = (idx << 1) | (uint32_t)((g >> op.q[b]) & 1ULL);
            const double2 d = pool[op.mat + idx];
            if (d.x == 1.0 && d.y == 0.0) continue;
            sm[tswz(o)] = cmul_x(d, sm[tswz(o)]);
          }
          break;
        }
        case T_SWAP: {
          // pairs (i: t1 = 1, t2 = 0) <-> (j = i ^ both); the CTA owning i does the pair
          const uint64_t b1 = 1ULL << op.t1, b2 = 1ULL << op.t2;
          const uint64_t fixed1 = op.ctrl | b1;  // bits that must be 1 in i
          const uint64_t gate = op.ctrl | b1 | b2;
          const uint64_t hi_one = fixed1 & ~lmask, hi_zero = b2 & ~lmask;
          if ((gbase & hi_one) != hi_one || (gbase & hi_zero) != 0) break;
          const uint64_t zmask = gate & lmask;
          const uint32_t count = L >> __popcll((long long)zmask);
          const uint32_t lo_one = (uint32_t)(fixed1 & lmask);
          for (uint32_t k = tid; k < count; k += THREADS) {
            uint32_t o = k;
            for (uint64_t mm = zmask; mm; mm &= mm - 1) o = ins0(o, (uint32_t)(__ffsll((long long)mm) - 1));
            o |= lo_one;
            const uint64_t gi = gbase | o, gj = gi ^ b1 ^ b2;
            double2* pi = sm + tswz(o);
            double2* pj = elem(gj);
            const double2 a = *pi, b = *pj;
            *pi = b;
            *pj = a;
          }
          break;
        }
        case T_DENSE: {
          const uint32_t kq = op.k, D = 1u << kq;
          uint64_t gm = 0;
          for (uint32_t b = 0; b < kq; ++b) gm |= 1ULL << op.q[b];
          if ((gbase & gm & ~lmask) != 0) break;  // group base must have the gate bits zero
          const uint64_t zmask = gm & lmask;
          const uint32_t count = L >> __popcll((long long)zmask);
          for (uint32_t k = tid; k < count; k += THREADS) {
            uint32_t o = k;
            for (uint64_t mm = zmask; mm; mm &= mm - 1) o = ins0(o, (uint32_t)(__ffsll((long long)mm) - 1));
            const uint64_t base = gbase | o;
            double2 v[32];
            double2* ptr[32];
            for (uint32_t j = 0; j < D; ++j) {
              uint64_t off = 0;
              for (uint32_t b = 0; b < kq; ++b)
                if ((j >> (kq - 1 - b)) & 1u) off |= 1ULL << op.q[b];
              ptr[j] = elem(base | off);
              v[j] = *ptr[j];
            }
            for (uint32_t r = 0; r < D; ++r) {
              double2 acc = make_double2(0.0, 0.0);
              for (uint32_t c = 0; c < D; ++c) {
                const double2 uu = pool[op.mat + r * D + c];
                if (uu.x != 0.0 || uu.y != 0.0) acc = cadd_x(acc, cmul_x(uu, v[c]));
              }
              *ptr[r] = acc;
            }
          }
          break;
        }
        case T_MEASURE:
        case T_RESET: {
          const uint32_t q = op.t1;
          const uint64_t qb = 1ULL << q;
          double part = 0.0;
          if (q < lb) {
            for (uint32_t k = tid; k < L / 2; k += THREADS)
              part = __dadd_rn(part, norm_sqr_x(sm[tswz(ins0(k, q) | (uint32_t)qb)]));
          } else if (gbase & qb) {
            for (uint32_t o = tid; o < L; o += THREADS) part = __dadd_rn(part, norm_sqr_x(sm[tswz(o)]));
          }
          const double cta = block_sum_all<THREADS>(part, red);
          if (tid == 0) red[40] = cta;
          if (C > 1) cl.sync(); else __syncthreads();
          if (tid == 0) {
            double p1 = 0.0;
            for (uint32_t r = 0; r < C; ++r) {
              const double* pr = (r == rank) ? red : cl.map_shared_rank(red, r);
              p1 = __dadd_rn(p1, pr[40]);
            }
            s_bcast[0] = p1;
            s_count[0] = s_count[1] = 0;
            if (hi - lo == 1) {
              const uint64_t shot = shot_at(lo);
              double rr;
              if (P.draws && draws < P.draw_stride) {
                rr = P.draws[shot * P.draw_stride + draws];
              } else {
                uint32_t key[8];
                seed_key_from_u64(pg.base_seed + shot, key);
                rr = chacha8_draw(key, draws);
              }
              if (rank == 0 && draws >= tk.draws && fabs(rr - p1) < 1e-12) atomicAdd(P.boundary, 1ULL);
              s_count[rr < p1 ? 1 : 0] = 1;
            }
          }
          __syncthreads();
          const double p1 = s_bcast[0];
          if (hi - lo > 1) {
            // each shot's own draw; outcome 0 goes to the front of the other
            // list, outcome 1 to its back
            const uint32_t dst = src == 0 ? 1 : 0;
            if (rank == 0) {
              for (uint32_t i = lo + tid; i < hi; i += THREADS) {
                const uint64_t shot = shot_at(i);
                double rr;
                if (P.draws && draws < P.draw_stride) {
                  rr = P.draws[shot * P.draw_stride + draws];
                } else {
                  uint32_t key[8];
                  seed_key_from_u64(pg.base_seed + shot, key);
                  rr = chacha8_draw(key, draws);
                }
                // (a program run again from the start draws what was counted before)
                if (draws >= tk.draws && fabs(rr - p1) < 1e-12) atomicAdd(P.boundary, 1ULL);
                if (rr < p1) P.order[dst][hi - 1 - atomicAdd(&s_count[1], 1u)] = (uint32_t)shot;
                else P.order[dst][lo + atomicAdd(&s_count[0], 1u)] = (uint32_t)shot;
              }
              __threadfence();
            }
            if (C > 1) cl.sync(); else __syncthreads();
            if (rank != 0 && tid == 0) {
              const uint32_t* c0 = cl.map_shared_rank(&s_count[0], 0);
              s_count[0] = c0[0];
              s_count[1] = c0[1];
            }
            __syncthreads();
            src = dst;
          }
          ++draws;
          const uint32_t n0 = s_count[0], n1 = s_count[1];
          const int o = n1 > n0 ? 1 : 0;  // go on with the longer list
          if (n0 && n1) {
            if (tid == 0 && rank == 0) {
              atomicAdd(P.queue + 2, 1ULL);
              s_task = atomicAdd(P.queue + 1, 1ULL);
            }
            if (C > 1) cl.sync(); else __syncthreads();
            const unsigned long long t = rank == 0 ? s_task : *cl.map_shared_rank(&s_task, 0);
            const bool saved = t < P.nslots;
            if (saved) {
              double2* d = P.slots + (t << pg.n) + gbase;
              for (uint32_t i = tid; i < L; i += THREADS) __stcg(d + i, sm[i]);
              if (rank == 0)
                for (uint32_t i = tid; i < pg.ncbits; i += THREADS) P.slot_cbits[t * pg.ncbits + i] = cb[i];
              __threadfence();
            }
            if (C > 1) cl.sync(); else __syncthreads();
            if (tid == 0 && rank == 0) {
              TTask w{};
              w.prog = it.prog;
              w.oi = oi;
              w.lo = o ? lo : lo + n0;
              w.hi = o ? lo + n0 : hi;
              w.src = src;
              w.slot = saved ? (int32_t)t : -1;
              w.outcome = o ? 0u : 1u;
              w.draws = (uint32_t)draws;
              w.p1 = p1;
              P.tasks[t] = w;
              st_release(P.ready + t, 1);
            }
            if (o) lo += n0; else hi = lo + n0;
          }
          if (op.type == T_RESET && o == 1) ++n1q;  // the flip
          collapse(op, o, norm_of(o, p1));
          // read by conditions after this op's closing barrier only
          if (tid == 0 && op.type == T_MEASURE) cb[op.cbit] = o;
          break;
        }
        case T_RPHASE: {
          // the next op.k ops act on the four local bits q[0..3] only: each
          // thread holds the 16 amplitudes of a group in registers and applies
          // them in program order (one shared-memory pass, one barrier)
          const uint32_t cnt = op.k;
          const uint32_t r0 = op.q[0], r1 = op.q[1], r2 = op.q[2], r3 = op.q[3];
          const uint32_t s0 = tswz(1u << r0), s1 = tswz(1u << r1), s2 = tswz(1u << r2),
                         s3 = tswz(1u << r3);
          auto sidx = [&](uint32_t sb, int j) {
            return sb ^ ((j & 1) ? s0 : 0u) ^ ((j & 2) ? s1 : 0u) ^ ((j & 4) ? s2 : 0u) ^
                   ((j & 8) ? s3 : 0u);
          };
          const uint32_t groups = L >> 4;
          for (uint32_t gi = tid; gi < groups; gi += THREADS) {
            // tswz is linear over XOR and the group base has the register bits clear
            const uint32_t sb = tswz(ins0(ins0(ins0(ins0(gi, r0), r1), r2), r3));
            double2 a[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) a[j] = sm[sidx(sb, j)];
            for (uint32_t sidx_op = 0; sidx_op < cnt; ++sidx_op) {
              const TOp so = ops[pg.ops_off + oi + 1 + sidx_op];
              if (gi == 0) (so.remote & kOpMulti ? nnq : n1q) += 1;
              const uint32_t t = so.t1;
              const uint32_t rt = t == r0 ? 0u : (t == r1 ? 1u : (t == r2 ? 2u : 3u));
              uint32_t creg = 0;
              if (so.ctrl) {
                if ((so.ctrl >> r0) & 1ULL) creg |= 1u;
                if ((so.ctrl >> r1) & 1ULL) creg |= 2u;
                if ((so.ctrl >> r2) & 1ULL) creg |= 4u;
                if ((so.ctrl >> r3) & 1ULL) creg |= 8u;
              }
              if (so.type == T_ONEQ) {
                double2 uu[4];
                for (int i = 0; i < 4; ++i) uu[i] = pool[so.mat + i];
                switch (rt) {
                  case 0: rphase_1q<0>(a, uu, creg); break;
                  case 1: rphase_1q<1>(a, uu, creg); break;
                  case 2: rphase_1q<2>(a, uu, creg); break;
                  default: rphase_1q<3>(a, uu, creg); break;
                }
              } else {
                switch (rt) {
                  case 0: rphase_x<0>(a, creg); break;
                  case 1: rphase_x<1>(a, creg); break;
                  case 2: rphase_x<2>(a, creg); break;
                  default: rphase_x<3>(a, creg); break;
                }
              }
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) sm[sidx(sb, j)] = a[j];
          }
          // continue after the phase's ops
          oi += cnt;
          if (oi + 1 < pg.nops) fetch(oi + 1);
          break;
        }
        case T_FAIL:
          if (tid == 0 && rank == 0) atomicMin(P.failed, ((long long)it.prog << 40) | op.inst);
          break;
        default:
          break;
      }
      sync_all(remote);
      last_cluster = remote || C == 1;
      if (op.type == T_FAIL) break;
    }
    // classical bits and (optionally) the final state out; the next
    // trajectory re-initialises after a cluster barrier
    if (rank == 0)
      for (uint64_t i = tid; i < (uint64_t)(hi - lo) * pg.ncbits; i += THREADS) {
        const uint32_t k = (uint32_t)(i / pg.ncbits), c = (uint32_t)(i - (uint64_t)k * pg.ncbits);
        P.cbits_out[pg.cbits_off + shot_at(lo + k) * pg.ncbits + c] = cb[c];
      }
    if (pg.state_out) {
      double2* dst = pg.state_out + (it.shot << pg.n) + gbase;
      for (uint32_t i = tid; i < L; i += THREADS) dst[i] = sm[tswz(i)];
    }
    if (pg.counts && rank == 0 && tid == 0) {
      pg.counts[0] = n1q;
      pg.counts[1] = nnq;
      pg.counts[2] = nmeas;
    }
    sync_all(true);
    if (rank == 0 && tid == 0) atomicAdd(P.queue + 2, ~0ULL);
  }
}

// ---- host side ---------------------------------------------------------------

struct Encoded {
  std::vector<TOp> ops;
  std::vector<double2> pool;
};

uint32_t push_mat(Encoded& e, const hc* m, uint32_t count) {
  const uint32_t off = (uint32_t)e.pool.size();
  for (uint32_t i = 0; i < count; ++i) e.pool.push_back(make_double2(m[i].re, m[i].im));
  return off;
}

TOp blank_op(int64_t inst, const dq_inst* in) {
  TOp t{};
  t.inst = inst;
  t.cbit = -1;
  if (in) {
    t.cond_first = in->cond_first;
    t.cond_count = in->cond_count;
  }
  return t;
}

void encode_gateop(Encoded& e, const GateOp& g, TOp t) {
  switch (g.cls) {
    case GC_ONE_Q:
      t.type = T_ONEQ;
      t.t1 = (uint8_t)g.target;
      t.ctrl = g.ctrl_mask;
      t.mat = push_mat(e, g.u, 4);
      break;
    case GC_PHASE:
      t.type = T_PHASE;
      t.t1 = (uint8_t)g.target;
      t.ctrl = g.ctrl_mask;
      t.mat = push_mat(e, g.u, 1);
      break;
    case GC_XPERM:
      t.type = T_XPERM;
      t.t1 = (uint8_t)g.target;
      t.ctrl = g.ctrl_mask;
      break;
    case GC_SWAP:
      t.type = T_SWAP;
      t.t1 = (uint8_t)g.target;
      t.t2 = (uint8_t)g.target2;
      t.ctrl = g.ctrl_mask;
      break;
    case GC_DIAG: {
      t.type = T_DIAG;
      t.k = (uint8_t)g.dense.k;
      for (uint32_t b = 0; b < g.dense.k; ++b) t.q[b] = (uint8_t)g.dense.qubits[b];
      const uint32_t D = 1u << g.dense.k;
      std::vector<hc> d(D);
      for (uint32_t i = 0; i < D; ++i) d[i] = g.dense.m[i * D + i];
      t.mat = push_mat(e, d.data(), D);
      break;
    }
    case GC_DENSE: {
      t.type = T_DENSE;
      t.k = (uint8_t)g.dense.k;
      for (uint32_t b = 0; b < g.dense.k; ++b) t.q[b] = (uint8_t)g.dense.qubits[b];
      const uint32_t D = 1u << g.dense.k;
      t.mat = push_mat(e, g.dense.m, D * D);
      break;
    }
    default:
      t.type = T_NOP;
      break;
  }
  e.ops.push_back(t);
}

// The shot program (fuse_program), or with DQ_SEM_SIMULATE the instructions one
// by one, as device ops, appended to e.
int encode_program(const dq_inst* prog, uint64_t ninst, uint32_t n, uint32_t cond_base,
                   Encoded& e, int semantics = DQ_SEM_SHOTS) {
  std::vector<FusedEntry> fused;
  if (semantics == DQ_SEM_SHOTS) {
    fused = fuse_program(prog, ninst, n);
  } else {
    fused.resize(ninst);
    for (uint64_t i = 0; i < ninst; ++i) fused[i].inst = (int64_t)i;
  }
  for (const FusedEntry& f : fused) {
    if (f.inst < 0) {
      GateOp g;
      classify_1q(f.m, f.qubit, 0, g);
      encode_gateop(e, g, blank_op(-1, nullptr));
      continue;
    }
    const dq_inst& in = prog[f.inst];
    TOp t = blank_op(f.inst, &in);
    t.cond_first += cond_base;
    switch (in.kind) {
      case DQ_ID: case DQ_U0: case DQ_BARRIER: case DQ_CLASSICAL: case DQ_G_NOOP:
        continue;
      case DQ_G_OPAQUE:  // a no-op in the shot path (run_instruction_par)
        if (semantics == DQ_SEM_SHOTS) continue;
        t.type = T_FAIL;
        e.ops.push_back(t);
        continue;
      case DQ_G_UNSUPPORTED:
        t.type = T_FAIL;
        e.ops.push_back(t);
        continue;
      case DQ_MEASURE:
        t.type = T_MEASURE;
        t.t1 = (uint8_t)in.q[0];
        t.cbit = (int32_t)in.cbit;
        e.ops.push_back(t);
        continue;
      case DQ_RESET:
        t.type = T_RESET;
        t.t1 = (uint8_t)in.q[0];
        e.ops.push_back(t);
        continue;
      default:
        break;
    }
    GateOp g;
    if (!inst_to_op(in, g)) return fail(DQ_ERR_INTERNAL, "instruction kind without a matrix");
    if (gate_qubit_count(in.kind) != 1) t.remote = kOpMulti;
    encode_gateop(e, g, t);
  }
  return DQ_OK;
}

void mark_remote(TOp* ops, size_t count, uint32_t lb) {
  const uint64_t lmask = (1ULL << lb) - 1;
  for (size_t i = 0; i < count; ++i) {
    TOp& t = ops[i];
    uint64_t touched = 0;
    switch (t.type) {
      case T_ONEQ: case T_XPERM: touched = 1ULL << t.t1; break;
      case T_SWAP: touched = (1ULL << t.t1) | (1ULL << t.t2); break;
      case T_DENSE:
        for (uint32_t b = 0; b < t.k; ++b) touched |= 1ULL << t.q[b];
        break;
      case T_MEASURE: case T_RESET: t.remote |= 1u; continue;
      default: break;
    }
    t.remote = (t.remote & kOpMulti) | ((touched & ~lmask) ? 1u : 0u);
  }
}

// Register phases: maximal runs (two or more) of unconditional T_ONEQ /
// T_XPERM ops whose targets and controls all lie within four local bits
// become one T_RPHASE header followed by the ops (in program order).
std::vector<TOp> group_phases(const std::vector<TOp>& ops, uint32_t lb) {
  std::vector<TOp> out;
  if (lb < 4) return ops;
  const uint64_t lmask = (1ULL << lb) - 1;
  auto bits_of = [](const TOp& t) { return t.ctrl | (1ULL << t.t1); };
  auto eligible = [&](const TOp& t) {
    return (t.type == T_ONEQ || t.type == T_XPERM) && t.cond_count == 0 && !(t.remote & 1u) &&
           (bits_of(t) & ~lmask) == 0;
  };
  size_t i = 0;
  while (i < ops.size()) {
    if (!eligible(ops[i])) {
      out.push_back(ops[i++]);
      continue;
    }
    uint64_t set = bits_of(ops[i]);
    size_t j = i + 1;
    while (j < ops.size() && j - i < 255 && eligible(ops[j]) &&
           __builtin_popcountll(set | bits_of(ops[j])) <= 4) {
      set |= bits_of(ops[j]);
      ++j;
    }
    if (j - i < 2 || __builtin_popcountll(set) > 4) {
      out.push_back(ops[i++]);
      continue;
    }
    for (uint32_t b = 0; b < lb && __builtin_popcountll(set) < 4; ++b) set |= 1ULL << b;
    TOp h{};
    h.type = T_RPHASE;
    h.k = (uint8_t)(j - i);
    h.inst = ops[i].inst;
    int nb = 0;
    for (uint32_t b = 0; b < lb; ++b)
      if ((set >> b) & 1ULL) h.q[nb++] = (uint8_t)b;
    out.push_back(h);
    for (size_t k = i; k < j; ++k) out.push_back(ops[k]);
    i = j;
  }
  return out;
}

// All programs and trajectories of one launch (one cluster span).
struct LaunchSet {
  Encoded enc;
  std::vector<dq_cond> conds;
  std::vector<TProg> progs;
  std::vector<TItem> items;
  // sweep programs of the HBM items, staged in pinned host memory
  const uint8_t* blob_host = nullptr;
  size_t blob_host_bytes = 0;
  std::vector<TSweep> sweeps;
  uint32_t C = 1;
  uint32_t max_lb = 1, max_ncbits = 0;
  size_t hbm_smem = 0;           // shared memory the HBM items' sweeps need
};

// Largest batch item that runs as HBM-resident fused sweeps inside the
// persistent launch (2^30 amplitudes = 16 GiB).
constexpr uint32_t kHbmItemMaxQubits = 30;
// Sweep geometry of HBM items: 8 thread bits (the 256-thread trajectory
// CTA), 4 register bits, tiles of 2^12 amplitudes (two tile buffers, the
// slot factors and the staged program fit one CTA's shared memory).
constexpr uint32_t kHbmTB = 8, kHbmM = kHbmTileBits;

// A unitary batch item planned as fused sweeps for the HBM path of k_traj.
struct HbmPlan {
  std::vector<uint8_t> blob;
  std::vector<uint64_t> offs;
  int64_t synth = -1;
  uint32_t perm[64];
};

// Plans item `it` (shot semantics, from |0...0>) as sweeps of the HBM
// geometry; false when the item has measurements, resets or conditions, or a
// gate the sweep planner does not represent (such items run on the engine).
bool plan_hbm_item(const dq_batch_item& it, HbmPlan* out) {
  for (uint64_t i = 0; i < it.ninst; ++i) {
    const dq_inst& in = it.prog[i];
    if (in.cond_count || in.kind == DQ_MEASURE || in.kind == DQ_RESET || in.kind == DQ_G_UNSUPPORTED)
      return false;
  }
  for (uint32_t l = 0; l < 64; ++l) out->perm[l] = l;
  uint32_t rb = 0;
  if (fused_plan(it.n, it.prog, it.ninst, DQ_SEM_SHOTS, kHbmTB, (int)kHbmM, 0, &out->blob, &out->offs,
                 out->perm, &out->synth, &rb) != DQ_OK ||
      (!out->offs.empty() && rb != kHbmM - kHbmTB)) {
    clear_error();
    return false;
  }
  return true;
}

// Adds a planned HBM item whose state lives at `hbm` (device, 2^n amplitudes)
// and whose sweep programs sit at byte `base` of the set's program blob.
void add_hbm_program(LaunchSet& ls, const HbmPlan& pl, uint64_t base, uint32_t n,
                     uint64_t cbits_off, uint32_t ncbits, double2* hbm) {
  TProg pg{};
  pg.n = n;
  pg.lb = 13;  // reported local bits; the HBM branch sizes its shared memory by hbm_smem
  pg.ncbits = ncbits;
  pg.cbits_off = cbits_off;
  pg.hbm = hbm;
  pg.sweep_first = (uint32_t)ls.sweeps.size();
  pg.nsweeps = (uint32_t)pl.offs.size();
  pg.synth = (long long)pl.synth;
  for (uint64_t off : pl.offs) {
    const uint32_t pb = sweep_prog_bytes(pl.blob.data() + off);
    ls.sweeps.push_back(TSweep{base + off, 1u << (n - kHbmM), sweep_run_bits(pl.blob.data() + off),
                               pb, sweep_flags(pl.blob.data() + off) & SWF_MICRO});
    ls.hbm_smem = std::max<size_t>(ls.hbm_smem, sizeof(double2) * (2 * (1u << kHbmM) + kMaxSlots) + pb);
  }
  ls.progs.push_back(pg);
  ls.max_lb = std::max(ls.max_lb, pg.lb);
  ls.max_ncbits = std::max(ls.max_ncbits, ncbits);
}

// Op types whose `mat` indexes the matrix pool (push_mat in encode_gateop).
bool op_uses_pool(uint8_t type) {
  return type == T_ONEQ || type == T_PHASE || type == T_DIAG || type == T_DENSE;
}

// One program's ops and matrices, encoded on its own (matrix offsets into
// its own pool, condition offsets from 0) so that programs can be encoded
// on several host threads and appended to a launch set afterwards.
struct ProgCode {
  std::vector<TOp> ops;
  std::vector<double2> pool;
  int rc = DQ_OK;
  std::string err;
};

void encode_prog_code(const dq_inst* prog, uint64_t ninst, uint32_t n, uint32_t lb, ProgCode& out) {
  Encoded e;
  out.rc = encode_program(prog, ninst, n, 0, e);
  if (out.rc != DQ_OK) {
    out.err = dq_last_error();
    return;
  }
  mark_remote(e.ops.data(), e.ops.size(), lb);
  out.ops = group_phases(e.ops, lb);
  out.pool = std::move(e.pool);
}

// Appends a program encoded by encode_prog_code: the same records add_program
// would write (matrix and condition offsets moved to the set's pools).
int add_prog_code(LaunchSet& ls, const ProgCode& pc, const dq_cond* conds, uint64_t nconds,
                  uint32_t n, uint32_t lb, uint64_t base_seed, uint64_t cbits_off, uint32_t ncbits,
                  double2* state_out) {
  if (pc.rc != DQ_OK) return fail(pc.rc, pc.err);
  TProg pg{};
  pg.ops_off = (uint32_t)ls.enc.ops.size();
  const uint32_t pool_base = (uint32_t)ls.enc.pool.size();
  const uint32_t cond_base = (uint32_t)ls.conds.size();
  for (uint64_t c = 0; c < nconds; ++c) ls.conds.push_back(conds[c]);
  ls.enc.pool.insert(ls.enc.pool.end(), pc.pool.begin(), pc.pool.end());
  for (TOp t : pc.ops) {
    if (op_uses_pool(t.type)) t.mat += pool_base;
    if (t.cond_count) t.cond_first += cond_base;
    ls.enc.ops.push_back(t);
  }
  pg.nops = (uint32_t)pc.ops.size();
  pg.n = n;
  pg.lb = lb;
  pg.ncbits = ncbits;
  pg.base_seed = base_seed;
  pg.cbits_off = cbits_off;
  pg.state_out = state_out;
  ls.progs.push_back(pg);
  ls.max_lb = std::max(ls.max_lb, lb);
  ls.max_ncbits = std::max(ls.max_ncbits, ncbits);
  return DQ_OK;
}

int add_program(LaunchSet& ls, const dq_inst* prog, uint64_t ninst, const dq_cond* conds,
                uint64_t nconds, uint32_t n, uint32_t lb, uint64_t base_seed, uint64_t cbits_off,
                uint32_t ncbits, double2* state_out) {
  TProg pg{};
  pg.ops_off = (uint32_t)ls.enc.ops.size();
  const uint32_t cond_base = (uint32_t)ls.conds.size();
  for (uint64_t c = 0; c < nconds; ++c) ls.conds.push_back(conds[c]);
  DQ_TRY(encode_program(prog, ninst, n, cond_base, ls.enc));
  pg.nops = (uint32_t)(ls.enc.ops.size() - pg.ops_off);
  mark_remote(ls.enc.ops.data() + pg.ops_off, pg.nops, lb);
  {
    const std::vector<TOp> tail(ls.enc.ops.begin() + pg.ops_off, ls.enc.ops.end());
    const std::vector<TOp> grouped = group_phases(tail, lb);
    ls.enc.ops.resize(pg.ops_off);
    ls.enc.ops.insert(ls.enc.ops.end(), grouped.begin(), grouped.end());
    pg.nops = (uint32_t)grouped.size();
  }
  pg.n = n;
  pg.lb = lb;
  pg.ncbits = ncbits;
  pg.base_seed = base_seed;
  pg.cbits_off = cbits_off;
  pg.state_out = state_out;
  ls.progs.push_back(pg);
  ls.max_lb = std::max(ls.max_lb, lb);
  ls.max_ncbits = std::max(ls.max_ncbits, ncbits);
  return DQ_OK;
}

// The shots of the set's only program: one item whose shots share states
// (shot indices of the lists are 32-bit; more shots than that run one by one).
void add_shots(LaunchSet& ls, uint64_t shots) {
  if (shots == 0) return;
  if (shots < (1ULL << 31)) {
    ls.items.push_back(TItem{0, (uint32_t)shots, 0});
    return;
  }
  ls.items.resize(shots);
  for (uint64_t s = 0; s < shots; ++s) ls.items[s] = TItem{0, 1, s};
}

// Launch geometry of k_traj: opt-in shared memory, cluster dimension and as
// many clusters as can be resident at once (capped by the item count).
struct TrajLaunch {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[1];
  int threads = 256;
  uint32_t clusters = 0;
};

template <int THREADS>
int config_traj_t(uint32_t C, size_t smem, uint64_t nitems, TrajLaunch* L) {
  DQ_TRY(allow_shared((const void*)k_traj<THREADS>, smem));
  L->attr[0].id = cudaLaunchAttributeClusterDimension;
  L->attr[0].val.clusterDim.x = C;
  L->attr[0].val.clusterDim.y = 1;
  L->attr[0].val.clusterDim.z = 1;
  L->cfg.blockDim = dim3(THREADS, 1, 1);
  L->cfg.dynamicSmemBytes = smem;
  L->cfg.attrs = L->attr;
  L->cfg.numAttrs = 1;
  L->cfg.gridDim = dim3(C, 1, 1);
  int max_clusters = 0;
  cudaError_t e = cudaOccupancyMaxActiveClusters(&max_clusters, (void*)k_traj<THREADS>, &L->cfg);
  if (e != cudaSuccess || max_clusters < 1) {
    cudaGetLastError();
    return fail(DQ_ERR_UNSUPPORTED, std::string("trajectory kernel does not fit: cluster of ") +
                                        std::to_string(C) + " CTAs x " + std::to_string(smem) +
                                        " B shared memory");
  }
  uint64_t ncl = std::min<uint64_t>((uint64_t)max_clusters, nitems);
  if (ncl < 1) ncl = 1;
  L->cfg.gridDim = dim3((unsigned)(ncl * C), 1, 1);
  L->threads = THREADS;
  L->clusters = (uint32_t)ncl;
  return DQ_OK;
}

int config_traj(int threads, uint32_t C, size_t smem, uint64_t nitems, TrajLaunch* L) {
  if (threads == 128) return config_traj_t<128>(C, smem, nitems, L);
  if (threads == 256) return config_traj_t<256>(C, smem, nitems, L);
  return config_traj_t<512>(C, smem, nitems, L);
}

int launch_traj(TrajLaunch& L, const TrajParams& P, cudaStream_t st) {
  L.cfg.stream = st;
  L.cfg.attrs = L.attr;
  if (L.threads == 128) DQ_CUDA_TRY(cudaLaunchKernelEx(&L.cfg, k_traj<128>, P));
  else if (L.threads == 256) DQ_CUDA_TRY(cudaLaunchKernelEx(&L.cfg, k_traj<256>, P));
  else DQ_CUDA_TRY(cudaLaunchKernelEx(&L.cfg, k_traj<512>, P));
  return DQ_OK;
}

size_t traj_smem(const LaunchSet& ls) {
  return std::max<size_t>(ls.hbm_smem, sizeof(double2) * (1u << ls.max_lb) + sizeof(double) * 48 +
                                           sizeof(int32_t) * std::max<uint32_t>(ls.max_ncbits, 1));
}

// Dynamic shared memory of a launch whose ops, pool and conds are one image of
// `image` bytes: with the image, when it is small next to the states.
size_t stage_tables(const LaunchSet& ls, TrajParams& P, size_t image) {
  const size_t base = (traj_smem(ls) + 15) / 16 * 16;
  if (ls.hbm_smem || image > 32 * 1024 || base + image > 220 * 1024) return traj_smem(ls);
  P.stage_bytes = (uint32_t)image;
  P.stage_at = (uint32_t)base;
  return base + image;
}

// Device buffers of one launch, freed on scope exit.
struct LaunchBuffers {
  TOp* ops = nullptr;
  double2* pool = nullptr;
  dq_cond* conds = nullptr;
  TProg* progs = nullptr;
  TItem* items = nullptr;
  unsigned long long* ctr = nullptr;  // [0..2] queue, [3] boundary, [4] failed
  void* share = nullptr;              // shot lists, tasks, draws and small states (set_shared)
  void* pooled_share = nullptr;       // the same for one launch, from the engine's pool
  void* slots = nullptr;              // saved states, from the engine's buffer cache
  size_t slot_bytes = 0;
  int device = 0;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  cudaStream_t st = nullptr;
  bool own_st = false;  // destroy st with the buffers
  void* block = nullptr;      // one launch's buffers, from the engine's pool on st
  void* stage = nullptr;      // their pinned image, if there is one
  size_t stage_bytes = 0;
  ~LaunchBuffers() {
    if (st) cudaStreamSynchronize(st);
    if (block) cudaFreeAsync(block, st);
    if (pooled_share) cudaFreeAsync(pooled_share, st);
    pinned_free(stage_bytes, stage);
    if (ops) cudaFree(ops);
    if (pool) cudaFree(pool);
    if (conds) cudaFree(conds);
    if (progs) cudaFree(progs);
    if (items) cudaFree(items);
    if (ctr) cudaFree(ctr);
    if (share) cudaFree(share);
    if (slots) cache_free(device, slot_bytes, slots);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    if (own_st && st) cudaStreamDestroy(st);
  }
};

template <class T>
int upload(T** dst, const std::vector<T>& v, cudaStream_t st) {
  const size_t bytes = sizeof(T) * std::max<size_t>(v.size(), 1);
  DQ_CUDA_TRY(cudaMalloc((void**)dst, bytes));
  if (!v.empty())
    DQ_CUDA_TRY(cudaMemcpyAsync(*dst, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice, st));
  return DQ_OK;
}

constexpr int kCtrWords = 5;
constexpr unsigned long long kNotFailed = 0x7fffffffffffffffULL;

uint32_t draws_of(const TOp* ops, size_t n) {
  uint32_t d = 0;
  for (size_t i = 0; i < n; ++i) d += ops[i].type == T_MEASURE || ops[i].type == T_RESET;
  return d;
}

// Buffers of a launch whose single program is shared by `shots` shots with up
// to `ndraws` draws each.  Saved states take at most 1 GiB (a split past that
// runs its program again from the start, as every shot would without sharing),
// the table of draws at most 64 MiB (draws past it are computed in place).
// DQ_ERR_OOM without memory for them, with b and P as they were.
// st: buffers from the engine's pool on that stream; null: they outlive a launch.
int set_shared(LaunchBuffers& b, TrajParams& P, int device, uint32_t n, uint64_t shots, uint32_t ncbits,
               uint32_t ndraws, cudaStream_t st) {
  if (shots < 2 || ndraws == 0) return DQ_OK;
  b.device = device;
  const size_t state = sizeof(double2) << n;
  uint64_t slots = shots - 1;
  const bool inline_slots = slots * state <= (64ULL << 20);
  if (!inline_slots) {  // powers of two: few sizes in the buffer cache
    slots = 1;
    while (slots < shots - 1 && 2 * slots * state <= (1ULL << 30)) slots *= 2;
    while (slots && cache_alloc(device, slots * state, &b.slots) != DQ_OK) {
      clear_error();
      b.slots = nullptr;
      slots /= 2;
    }
    b.slot_bytes = slots * state;
  }
  const uint32_t blocks = (ndraws + 7) / 8;
  const bool table = shots * blocks * 64 <= (64ULL << 20);
  size_t off[7], at = 0;
  const size_t bytes[6] = {4 * shots, 4 * shots, sizeof(TTask) * shots, 4 * (size_t)slots * ncbits,
                           table ? (size_t)shots * blocks * 64 : 0, inline_slots ? slots * state : 0};
  for (int i = 0; i < 6; ++i) {
    off[i] = at;
    at += (bytes[i] + 15) / 16 * 16;
  }
  off[6] = at;  // ready flags
  void** mem = st ? &b.pooled_share : &b.share;
  const size_t need = at + 4 * shots;
  const cudaError_t e = st ? pool_malloc_async(mem, need, st)
                           : alloc_refused(need) ? cudaErrorMemoryAllocation : cudaMalloc(mem, need);
  if (e != cudaSuccess) {
    cudaGetLastError();
    *mem = nullptr;
    if (b.slots) cache_free(device, b.slot_bytes, b.slots);
    b.slots = nullptr;
    return fail(e == cudaErrorMemoryAllocation ? DQ_ERR_OOM : DQ_ERR_CUDA,
                std::string("shared shots: ") + cudaGetErrorString(e));
  }
  uint8_t* base = static_cast<uint8_t*>(*mem);
  P.order[0] = reinterpret_cast<uint32_t*>(base + off[0]);
  P.order[1] = reinterpret_cast<uint32_t*>(base + off[1]);
  P.tasks = reinterpret_cast<TTask*>(base + off[2]);
  P.slot_cbits = reinterpret_cast<int32_t*>(base + off[3]);
  P.draws = table ? reinterpret_cast<double*>(base + off[4]) : nullptr;
  P.draw_stride = blocks * 8;
  P.ready = reinterpret_cast<int*>(base + off[6]);
  P.slots = inline_slots ? reinterpret_cast<double2*>(base + off[5]) : static_cast<double2*>(b.slots);
  P.nslots = (uint32_t)slots;
  return DQ_OK;
}

// set_shared, or without memory for it an item of its own for every shot.
int share_or_split(LaunchSet& ls, LaunchBuffers& b, TrajParams& P, int device, cudaStream_t st) {
  if (ls.items.size() != 1 || ls.items[0].count < 2) return DQ_OK;
  const uint64_t shots = ls.items[0].count;
  const int rc = set_shared(b, P, device, ls.progs[0].n, shots, ls.progs[0].ncbits,
                            draws_of(ls.enc.ops.data(), ls.enc.ops.size()), st);
  if (rc != DQ_ERR_OOM) return rc;
  clear_error();
  ls.items.resize(shots);
  for (uint64_t s = 0; s < shots; ++s) ls.items[s] = TItem{0, 1, s};
  return DQ_OK;
}

// Work enqueued before every launch of a set_shared program.
int reset_shared(const TrajParams& P, uint64_t shots, cudaStream_t st) {
  if (!P.tasks) return DQ_OK;
  DQ_CUDA_TRY(cudaMemsetAsync(P.ready, 0, 4 * shots, st));
  if (P.draws) {
    const uint64_t work = shots * (P.draw_stride / 8);
    k_traj_draws<<<(unsigned)((work + 127) / 128), 128, 0, st>>>(P.progs, shots, P.draw_stride / 8,
                                                                  const_cast<double*>(P.draws));
    DQ_CUDA_TRY(cudaGetLastError());
  }
  return DQ_OK;
}

// Runs every item of ls in one persistent launch; cbits land in d_cbits.
int run_launch(LaunchSet& ls, int threads, int device, cudaStream_t st, int32_t* d_cbits,
               dq_traj_stats* acc) {
  if (ls.items.empty()) return DQ_OK;
  if (ls.enc.pool.empty()) ls.enc.pool.push_back(make_double2(0, 0));
  std::vector<uint8_t> pageable;  // the tables' image without pinned memory (outlives b's stream wait)
  LaunchBuffers b;
  b.st = st;
  // several shots of one program share states
  TrajParams P{};
  const uint64_t shots = ls.items.size() == 1 ? ls.items[0].count : 1;
  DQ_TRY(share_or_split(ls, b, P, device, st));
  // one allocation and one copy from pinned memory; the sweep programs of HBM
  // items are already pinned and follow in a copy of their own
  const unsigned long long init[kCtrWords] = {0ULL, 0ULL, ls.items.size(), 0ULL, kNotFailed};
  struct { const void* p; size_t bytes, off; } part[7] = {
      {ls.enc.ops.data(), sizeof(TOp) * ls.enc.ops.size(), 0},
      {ls.enc.pool.data(), sizeof(double2) * ls.enc.pool.size(), 0},
      {ls.conds.data(), sizeof(dq_cond) * ls.conds.size(), 0},
      {ls.progs.data(), sizeof(TProg) * ls.progs.size(), 0},
      {ls.items.data(), sizeof(TItem) * ls.items.size(), 0},
      {ls.sweeps.data(), sizeof(TSweep) * ls.sweeps.size(), 0},
      {init, sizeof(init), 0}};
  size_t image = 0;
  for (auto& x : part) {
    x.off = image;
    image += (x.bytes + 15) / 16 * 16;
  }
  if (pinned_alloc(image, &b.stage) == DQ_OK) {
    b.stage_bytes = image;
  } else {
    clear_error();
    pageable.resize(image);
  }
  uint8_t* stage = b.stage ? static_cast<uint8_t*>(b.stage) : pageable.data();
  for (const auto& x : part)
    if (x.bytes) memcpy(stage + x.off, x.p, x.bytes);
  DQ_CUDA_TRY(pool_malloc_async(&b.block, image + ls.blob_host_bytes, st));
  uint8_t* dev = static_cast<uint8_t*>(b.block);
  DQ_CUDA_TRY(cudaMemcpyAsync(dev, stage, image, cudaMemcpyHostToDevice, st));
  if (ls.blob_host_bytes)
    DQ_CUDA_TRY(cudaMemcpyAsync(dev + image, ls.blob_host, ls.blob_host_bytes, cudaMemcpyHostToDevice, st));
  unsigned long long* d_ctr = reinterpret_cast<unsigned long long*>(dev + part[6].off);
  DQ_CUDA_TRY(cudaEventCreate(&b.e0));
  DQ_CUDA_TRY(cudaEventCreate(&b.e1));
  P.ops = reinterpret_cast<const TOp*>(dev);
  P.pool = reinterpret_cast<const double2*>(dev + part[1].off);
  P.conds = reinterpret_cast<const dq_cond*>(dev + part[2].off);
  P.progs = reinterpret_cast<const TProg*>(dev + part[3].off);
  P.items = reinterpret_cast<const TItem*>(dev + part[4].off);
  P.sweeps = reinterpret_cast<const TSweep*>(dev + part[5].off);
  P.sweep_blob = dev + image;
  P.cbits_out = d_cbits;
  P.queue = d_ctr;
  P.boundary = d_ctr + 3;
  P.failed = reinterpret_cast<long long*>(d_ctr + 4);
  P.nitems = ls.items.size();
  TrajLaunch L;
  DQ_TRY(config_traj(threads, ls.C, stage_tables(ls, P, part[3].off), P.tasks ? shots : P.nitems, &L));
  const uint32_t clusters = L.clusters;
  DQ_CUDA_TRY(cudaEventRecord(b.e0, st));
  DQ_TRY(reset_shared(P, shots, st));
  DQ_TRY(launch_traj(L, P, st));
  DQ_CUDA_TRY(cudaEventRecord(b.e1, st));
  // into the staged image, whose copy has been consumed by then
  const unsigned long long* ctr = reinterpret_cast<const unsigned long long*>(stage);
  DQ_CUDA_TRY(cudaMemcpyAsync(stage, d_ctr, sizeof(init), cudaMemcpyDeviceToHost, st));
  DQ_CUDA_TRY(cudaStreamSynchronize(st));
  float ms = 0.f;
  DQ_CUDA_TRY(cudaEventElapsedTime(&ms, b.e0, b.e1));
  acc->boundary_draws += ctr[3];
  const long long f = (long long)ctr[4];
  if (f != 0x7fffffffffffffffLL && (acc->failed_inst < 0 || f < acc->failed_inst))
    acc->failed_inst = f;
  acc->kernel_ms += ms;
  acc->cluster_span = std::max(acc->cluster_span, ls.C);
  acc->clusters = clusters;
  acc->threads = (uint32_t)threads;
  acc->local_bits = std::max(acc->local_bits, ls.max_lb);
  acc->launches += 1;
  return DQ_OK;
}

int check_opts(const dq_traj_opts* opts, int* threads, uint32_t* max_span, uint32_t* force_lb) {
  dq_traj_opts o{};
  if (opts) o = *opts;
  *threads = o.threads ? o.threads : 256;
  if (*threads != 128 && *threads != 256 && *threads != 512)
    return fail(DQ_ERR_INVALID_ARG, "threads must be 128, 256 or 512");
  *max_span = o.max_cluster ? (uint32_t)o.max_cluster : 8u;
  if (*max_span != 1 && *max_span != 2 && *max_span != 4 && *max_span != 8)
    return fail(DQ_ERR_INVALID_ARG, "max_cluster must be 1, 2, 4 or 8");
  *force_lb = 0;
  if (o.local_bits) {
    if (o.local_bits < 1 || (uint32_t)o.local_bits > kLocalBitsMax)
      return fail(DQ_ERR_INVALID_ARG, "local_bits must be in 1..13");
    *force_lb = (uint32_t)o.local_bits;
  }
  return DQ_OK;
}

// Amplitudes per CTA (2^lb) and cluster span for an n-qubit trajectory.
int geometry(uint32_t n, uint32_t max_span, uint32_t force_lb, uint32_t* lb, uint32_t* C) {
  *lb = std::min(n, force_lb ? force_lb : kLocalBitsMax);
  // a smaller max_span needs more amplitudes per CTA than 2^13: not possible
  *C = 1u << (n - *lb);
  if (*C > max_span)
    return fail(DQ_ERR_INVALID_ARG, "a " + std::to_string(n) + "-qubit trajectory needs " +
                                        std::to_string(*C) + " CTAs per cluster, more than max_cluster");
  return DQ_OK;
}

// One program on a handle's state in a single launch of one CTA (k_traj): gates,
// measurements, resets and conditions with the state in shared memory.  Bound by
// the latency of one op after another; launching every gate and reading every
// p1 back costs about 3 us a gate and 20 us a measurement instead.
template <int THREADS>
int launch_small(size_t smem, const TrajParams& P, cudaStream_t st) {
  DQ_TRY(allow_shared((const void*)k_traj<THREADS>, smem));
  k_traj<THREADS><<<1, THREADS, smem, st>>>(P);
  DQ_CUDA_TRY(cudaGetLastError());
  return DQ_OK;
}

double ms_since(std::chrono::steady_clock::time_point t0) {
  return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
}

void init_stats(dq_traj_stats* s) {
  memset(s, 0, sizeof(*s));
  s->failed_inst = -1;
}

}  // namespace
}  // namespace dq

namespace dq {

// See dq_handle.cuh.  The handle's state is canonical or a pending basis state.
int small_run(dq_state_t h, const dq_inst* prog, uint64_t ninst, const dq_cond* conds, uint64_t nconds,
              uint64_t seed, int32_t* cbits, uint64_t ncbits, int semantics, dq_profile* prof) {
  Encoded e;
  DQ_TRY(encode_program(prog, ninst, h->n, 0, e, semantics));
  mark_remote(e.ops.data(), e.ops.size(), h->n);
  const std::vector<TOp> ops = group_phases(e.ops, h->n);
  TProg pg{};
  pg.nops = (uint32_t)ops.size();
  pg.n = pg.lb = h->n;
  pg.ncbits = (uint32_t)ncbits;
  pg.base_seed = seed;
  pg.state_out = h->amp;
  if (h->lazy_basis >= 0) pg.basis = (uint64_t)h->lazy_basis;
  else pg.state_in = h->amp;
  const TItem item{0, 1, 0};
  // one image up: tables, then the words that come back (counters, counts, bits)
  constexpr size_t kBack = sizeof(unsigned long long) * (kCtrWords + 3);
  const uint32_t ndraws = std::min<uint32_t>(draws_of(ops.data(), ops.size()), 4096);  // later ones in the kernel
  const size_t part[6] = {sizeof(TOp) * ops.size(), sizeof(double2) * e.pool.size(), sizeof(dq_cond) * nconds,
                          sizeof(TProg), sizeof(TItem), sizeof(double) * ndraws};
  size_t off[7], at = 0;
  for (int i = 0; i < 6; ++i) {
    off[i] = at;
    at += (part[i] + 15) / 16 * 16;
  }
  off[6] = at;
  const size_t back = kBack + sizeof(int32_t) * ncbits, bytes = at + back;
  DQ_TRY(ensure_query_buffers(h, bytes, bytes));
  uint8_t* up = static_cast<uint8_t*>(h->q_host);
  uint8_t* dev = static_cast<uint8_t*>(h->q_dev);
  unsigned long long* d_ctr = reinterpret_cast<unsigned long long*>(dev + off[6]);
  pg.counts = d_ctr + kCtrWords;
  pg.cbits_in = reinterpret_cast<const int32_t*>(dev + off[6] + kBack);
  const unsigned long long ctr[kCtrWords + 3] = {0, 0, 1, 0, kNotFailed, 0, 0, 0};
  const void* src[5] = {ops.data(), e.pool.data(), conds, &pg, &item};
  for (int i = 0; i < 5; ++i)
    if (part[i]) memcpy(up + off[i], src[i], part[i]);
  Chacha8Cursor rng;
  rng.seed(seed);
  for (uint32_t i = 0; i < ndraws; ++i) reinterpret_cast<double*>(up + off[5])[i] = rng.draw();
  memcpy(up + off[6], ctr, kBack);
  if (ncbits) memcpy(up + off[6] + kBack, cbits, sizeof(int32_t) * ncbits);
  DQ_CUDA_TRY(cudaMemcpyAsync(dev, up, bytes, cudaMemcpyHostToDevice, h->stream));
  TrajParams P{};
  P.ops = reinterpret_cast<const TOp*>(dev);
  P.pool = reinterpret_cast<const double2*>(dev + off[1]);
  P.conds = reinterpret_cast<const dq_cond*>(dev + off[2]);
  P.progs = reinterpret_cast<const TProg*>(dev + off[3]);
  P.items = reinterpret_cast<const TItem*>(dev + off[4]);
  P.cbits_out = reinterpret_cast<int32_t*>(dev + off[6] + kBack);
  P.queue = d_ctr;
  P.boundary = d_ctr + 3;
  P.failed = reinterpret_cast<long long*>(d_ctr + 4);
  P.nitems = 1;
  P.draws = ndraws ? reinterpret_cast<const double*>(dev + off[5]) : nullptr;
  P.draw_stride = ndraws;
  LaunchSet ls;
  ls.max_lb = h->n;
  ls.max_ncbits = (uint32_t)ncbits;
  const size_t smem = stage_tables(ls, P, off[3]);
  DQ_TRY(h->n <= 8 ? launch_small<128>(smem, P, h->stream) : launch_small<256>(smem, P, h->stream));
  h->lazy_basis = -1;  // the kernel writes the state, also up to a failing gate
  DQ_CUDA_TRY(cudaMemcpyAsync(up + off[6], dev + off[6], back, cudaMemcpyDeviceToHost, h->stream));
  DQ_CUDA_TRY(cudaStreamSynchronize(h->stream));
  unsigned long long got[kCtrWords + 3];
  memcpy(got, up + off[6], kBack);
  if (ncbits) memcpy(cbits, up + off[6] + kBack, sizeof(int32_t) * ncbits);
  prof->kernel_launches += 1;
  prof->boundary_draws += got[3];
  prof->apply_one_qubit_calls += got[kCtrWords];
  prof->apply_n_qubit_calls += got[kCtrWords + 1];
  prof->measure_qubit_calls += got[kCtrWords + 2];
  if (got[4] != kNotFailed) {
    prof->failed_inst = (int64_t)(got[4] & ((1ULL << 40) - 1));
    return fail(DQ_ERR_UNSUPPORTED, "unsupported generic gate");
  }
  return DQ_OK;
}

}  // namespace dq

// A trajectory batch captured once as a CUDA graph (seed upload, counter
// reset, the persistent launch, result copies) and replayed per call.
struct dq_traj_plan_s {
  int device = 0;
  uint64_t shots = 0, ncbits = 0;
  dq::LaunchBuffers buf;
  int32_t* d_cbits = nullptr;
  int32_t* h_cbits = nullptr;            // pinned
  uint64_t* h_seed = nullptr;            // pinned: base seed of the next replay
  unsigned long long* h_ctr = nullptr;   // pinned: kCtrWords initial, then kCtrWords results
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  dq::TrajLaunch L;
  dq::TrajParams P{};
  dq_traj_stats geom{};
  ~dq_traj_plan_s() {
    if (buf.st) cudaStreamSynchronize(buf.st);
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    if (d_cbits) cudaFree(d_cbits);
    if (h_cbits) cudaFreeHost(h_cbits);
    if (h_seed) cudaFreeHost(h_seed);
    if (h_ctr) cudaFreeHost(h_ctr);
  }
};

using namespace dq;

extern "C" {

int dq_run_trajectories(int device, uint32_t n, const dq_inst* prog, uint64_t ninst,
                        const dq_cond* conds, uint64_t nconds, uint64_t base_seed, uint64_t shot0,
                        uint64_t shots, int32_t* cbits_out, uint64_t ncbits,
                        const dq_traj_opts* opts, dq_traj_stats* stats) {
  dq_traj_stats acc;
  init_stats(&acc);
  if (stats) *stats = acc;
  if (n < 1 || n > kTrajMaxQubits)
    return fail(DQ_ERR_INVALID_ARG, "dq_run_trajectories: n must be in 1..16");
  if (ninst && !prog) return fail(DQ_ERR_INVALID_ARG, "null program");
  if (shots && ncbits && !cbits_out) return fail(DQ_ERR_INVALID_ARG, "null cbits output");
  if (ncbits > kTrajMaxCbits) return fail(DQ_ERR_INVALID_ARG, "at most 1024 classical bits");
  if (shots > (1ULL << 40)) return fail(DQ_ERR_INVALID_ARG, "too many shots");
  for (uint64_t i = 0; i < ninst; ++i) DQ_TRY(validate_inst(prog[i], n, nconds, ncbits, conds, i));
  int threads;
  uint32_t max_span, force_lb, lb, C;
  DQ_TRY(check_opts(opts, &threads, &max_span, &force_lb));
  DQ_TRY(geometry(n, max_span, force_lb, &lb, &C));
  const auto t0 = std::chrono::steady_clock::now();
  LaunchSet ls;
  ls.C = C;
  DQ_TRY(add_program(ls, prog, ninst, conds, nconds, n, lb, base_seed + shot0, 0,
                     (uint32_t)ncbits, nullptr));
  add_shots(ls, shots);
  acc.prepare_ms = ms_since(t0);

  DeviceGuard g(device);
  cudaStream_t st = nullptr;
  DQ_TRY(stream_take(device, &st));
  int32_t* d_out = nullptr;
  const size_t out_bytes = sizeof(int32_t) * (size_t)shots * ncbits;
  int rc = DQ_OK;
  cudaError_t e = pool_malloc_async((void**)&d_out, std::max<size_t>(out_bytes, 4), st);
  if (e != cudaSuccess) rc = fail(DQ_ERR_OOM, std::string("cudaMalloc(cbits): ") + cudaGetErrorString(e));
  if (rc == DQ_OK) rc = run_launch(ls, threads, device, st, d_out, &acc);
  if (rc == DQ_OK && out_bytes) {
    e = cudaMemcpyAsync(cbits_out, d_out, out_bytes, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) rc = fail(DQ_ERR_CUDA, std::string("copy cbits: ") + cudaGetErrorString(e));
  }
  if (d_out) cudaFreeAsync(d_out, st);
  stream_give(device, st);
  if (acc.failed_inst >= 0) acc.failed_inst &= (1LL << 40) - 1;
  if (stats) *stats = acc;
  DQ_TRY(rc);
  if (acc.failed_inst >= 0)
    return fail(DQ_ERR_UNSUPPORTED, "instruction " + std::to_string(acc.failed_inst) +
                                        ": unsupported generic gate reached in a trajectory");
  return DQ_OK;
}

int dq_run_batch(int device, const dq_batch_item* items, uint64_t nitems,
                 const dq_traj_opts* opts, dq_traj_stats* stats) {
  dq_traj_stats acc;
  init_stats(&acc);
  if (stats) *stats = acc;
  if (nitems && !items) return fail(DQ_ERR_INVALID_ARG, "null items");
  int threads;
  uint32_t max_span, force_lb;
  DQ_TRY(check_opts(opts, &threads, &max_span, &force_lb));
  for (uint64_t k = 0; k < nitems; ++k) {
    const dq_batch_item& it = items[k];
    const std::string pre = "item " + std::to_string(k) + ": ";
    if (it.n < 1 || it.n > kMaxQubits) return fail(DQ_ERR_INVALID_ARG, pre + "n must be in 1..34");
    if (it.ninst && !it.prog) return fail(DQ_ERR_INVALID_ARG, pre + "null program");
    if (it.ncbits && !it.cbits_out) return fail(DQ_ERR_INVALID_ARG, pre + "null cbits output");
    if (it.ncbits > kTrajMaxCbits) return fail(DQ_ERR_INVALID_ARG, pre + "at most 1024 classical bits");
    for (uint64_t i = 0; i < it.ninst; ++i) {
      const int rc = validate_inst(it.prog[i], it.n, it.nconds, it.ncbits, it.conds, i);
      if (rc != DQ_OK) return fail(rc, pre + dq_last_error());
    }
  }
  DeviceGuard g(device);
  const auto t0 = std::chrono::steady_clock::now();
  // DQSIM_BATCH_TIMING=1: host phase times on stderr
  static const bool timing = [] {
    const char* e = getenv("DQSIM_BATCH_TIMING");
    return e && atoi(e) != 0;
  }();
  auto tlast = t0;
  auto mark = [&](const char* what) {
    if (!timing) return;
    const auto now = std::chrono::steady_clock::now();
    fprintf(stderr, "[dq_run_batch] %-14s %8.3f ms\n", what,
            std::chrono::duration<double, std::milli>(now - tlast).count());
    tlast = now;
  };
  // One persistent launch takes every item it can: states of up to 16 qubits
  // live in a cluster's shared memory; unitary items of 17..30 qubits keep
  // their state in HBM and run as fused tile sweeps by one cluster each.
  // Everything shares one cluster span (the widest any item needs).  Left
  // for separate launches: items whose slice at that span would hold fewer
  // than 16 amplitudes, and every resident item when local_bits is forced
  // (grouped by span); left for the engine (one dq_run each): large items
  // with measurements, resets or conditions.
  std::vector<uint64_t> resident, hbm_items, engine_items, large;
  std::vector<HbmPlan> plans;
  for (uint64_t k = 0; k < nitems; ++k) {
    if (items[k].n <= kTrajMaxQubits) resident.push_back(k);
    else large.push_back(k);
  }
  {
    // plan the large items on host threads
    std::vector<HbmPlan> lp(large.size());
    std::vector<char> ok(large.size(), 0);
    const bool hbm_ok = threads == 256 && !force_lb;
    const unsigned hw = std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
    const unsigned nt = (unsigned)std::max<size_t>(1, std::min<size_t>(hw, large.size()));
    auto work = [&](unsigned t) {
      for (size_t i = t; i < large.size(); i += nt) {
        const dq_batch_item& it = items[large[i]];
        ok[i] = hbm_ok && it.n <= kHbmItemMaxQubits && plan_hbm_item(it, &lp[i]);
      }
    };
    std::vector<std::thread> th;
    for (unsigned t = 1; t < nt; ++t) th.emplace_back(work, t);
    work(0);
    for (auto& x : th) x.join();
    for (size_t i = 0; i < large.size(); ++i) {
      if (ok[i]) {
        hbm_items.push_back(large[i]);
        plans.push_back(std::move(lp[i]));
      } else {
        engine_items.push_back(large[i]);
      }
    }
  }
  mark("plan large");
  uint32_t Cmain = hbm_items.empty() ? 1u : std::min<uint32_t>(8u, max_span);
  for (uint64_t k : resident) {
    uint32_t lb, C;
    DQ_TRY(geometry(items[k].n, max_span, force_lb, &lb, &C));
    if (!force_lb) Cmain = std::max(Cmain, C);
  }
  const uint32_t cbits_main = (uint32_t)__builtin_ctz(Cmain);
  // set 0: the main launch (span Cmain); sets 1..4: spans 1, 2, 4, 8 for the rest
  LaunchSet sets[5];
  sets[0].C = Cmain;
  for (int c = 0; c < 4; ++c) sets[1 + c].C = 1u << c;
  std::vector<std::vector<uint64_t>> members(5);
  std::vector<uint32_t> item_lb(nitems, 0);
  for (uint64_t k : resident) {
    const uint32_t n = items[k].n;
    uint32_t lb, C;
    geometry(n, max_span, force_lb, &lb, &C);
    if (!force_lb && n >= cbits_main + 4) {
      item_lb[k] = n - cbits_main;
      members[0].push_back(k);
    } else {
      item_lb[k] = lb;
      members[1 + __builtin_ctz(C)].push_back(k);
    }
  }
  for (uint64_t h = 0; h < hbm_items.size(); ++h) members[0].push_back(hbm_items[h]);
  std::vector<int64_t> plan_of(nitems, -1);
  for (uint64_t h = 0; h < hbm_items.size(); ++h) plan_of[hbm_items[h]] = (int64_t)h;
  // HBM item states: one device allocation
  std::vector<uint64_t> hbm_off(hbm_items.size(), 0);
  uint64_t hbm_amps = 0;
  for (uint64_t h = 0; h < hbm_items.size(); ++h) {
    hbm_off[h] = hbm_amps;
    hbm_amps += 1ULL << items[hbm_items[h]].n;
  }
  // per set: state outputs packed into one device buffer, cbits likewise
  struct Out { uint64_t item, state_off, cbits_off; };
  std::vector<Out> outs[5];
  uint64_t state_amps[5] = {0, 0, 0, 0, 0}, cbit_words[5] = {0, 0, 0, 0, 0};
  for (int c = 0; c < 5; ++c) {
    // costliest first (longest-processing-time order for the work queue)
    std::vector<uint64_t>& m = members[c];
    std::stable_sort(m.begin(), m.end(), [&](uint64_t a, uint64_t b) {
      return (items[a].ninst << items[a].n) > (items[b].ninst << items[b].n);
    });
    for (uint64_t k : m) {
      const bool packed = items[k].state_out && plan_of[k] < 0;
      Out o{k, packed ? state_amps[c] : ~0ULL, cbit_words[c]};
      if (packed) state_amps[c] += 1ULL << items[k].n;
      cbit_words[c] += items[k].ncbits;
      outs[c].push_back(o);
    }
  }
  // encode the resident items on host threads (each into its own ops and
  // matrix pool; appended to the launch sets in queue order below)
  std::vector<ProgCode> codes(nitems);
  {
    std::vector<uint64_t> todo;
    for (int c = 0; c < 5; ++c)
      for (const Out& o : outs[c])
        if (plan_of[o.item] < 0) todo.push_back(o.item);
    const unsigned hw = std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
    const unsigned nt = (unsigned)std::max<size_t>(1, std::min<size_t>(hw, todo.size() / 8 + 1));
    auto work = [&](unsigned t) {
      for (size_t i = t; i < todo.size(); i += nt) {
        const uint64_t k = todo[i];
        encode_prog_code(items[k].prog, items[k].ninst, items[k].n, item_lb[k], codes[k]);
      }
    };
    std::vector<std::thread> th;
    for (unsigned t = 1; t < nt; ++t) th.emplace_back(work, t);
    work(0);
    for (auto& x : th) x.join();
  }
  // the HBM items' sweep programs, copied on host threads into one pinned
  // staging buffer (recycled across calls) and uploaded with one copy
  std::vector<uint64_t> hbm_blob_off(plans.size(), 0);
  size_t hbm_blob_bytes = 0;
  for (size_t h = 0; h < plans.size(); ++h) {
    hbm_blob_off[h] = hbm_blob_bytes;
    hbm_blob_bytes += (plans[h].blob.size() + 15) / 16 * 16;
  }
  // returned to the pool on every exit path; each set's copies are complete
  // by then (run_launch synchronizes its stream, on errors too)
  struct PinnedStage {
    size_t bytes = 0;
    void* p = nullptr;
    ~PinnedStage() { pinned_free(bytes, p); }
  } stage;
  void* hbm_blob = nullptr;
  if (hbm_blob_bytes) {
    DQ_TRY(pinned_alloc(hbm_blob_bytes, &hbm_blob));
    stage.bytes = hbm_blob_bytes;
    stage.p = hbm_blob;
    const unsigned hw = std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
    const unsigned nt = (unsigned)std::max<size_t>(1, std::min<size_t>(hw, plans.size() / 8 + 1));
    auto work = [&](unsigned t) {
      for (size_t h = t; h < plans.size(); h += nt)
        memcpy(static_cast<uint8_t*>(hbm_blob) + hbm_blob_off[h], plans[h].blob.data(), plans[h].blob.size());
    };
    std::vector<std::thread> th;
    for (unsigned t = 1; t < nt; ++t) th.emplace_back(work, t);
    work(0);
    for (auto& x : th) x.join();
    sets[0].blob_host = static_cast<const uint8_t*>(hbm_blob);
    sets[0].blob_host_bytes = hbm_blob_bytes;
  }
  acc.prepare_ms = ms_since(t0);
  mark("group+encode");

  cudaStream_t st = nullptr;
  DQ_TRY(stream_take(device, &st));
  int rc = DQ_OK;
  double2* d_hbm = nullptr;
  if (hbm_amps) {
    // from the engine's size-keyed buffer cache: a repeated batch does not
    // pay cudaMalloc/cudaFree of its HBM states
    void* p = nullptr;
    rc = cache_alloc(device, sizeof(double2) * hbm_amps, &p);
    d_hbm = (double2*)p;
  }
  for (int c = 0; c < 5 && rc == DQ_OK; ++c) {
    if (outs[c].empty()) continue;
    double2* d_states = nullptr;
    int32_t* d_cbits = nullptr;
    cudaError_t e = pool_malloc_async((void**)&d_states, sizeof(double2) * std::max<uint64_t>(state_amps[c], 1), st);
    if (e == cudaSuccess)
      e = pool_malloc_async((void**)&d_cbits, sizeof(int32_t) * std::max<uint64_t>(cbit_words[c], 1), st);
    if (e != cudaSuccess) rc = fail(DQ_ERR_OOM, std::string("cudaMalloc(batch outputs): ") + cudaGetErrorString(e));
    const auto tp = std::chrono::steady_clock::now();
    LaunchSet& ls = sets[c];
    for (const Out& o : outs[c]) {
      if (rc != DQ_OK) break;
      const dq_batch_item& it = items[o.item];
      const uint32_t pi = (uint32_t)ls.progs.size();
      if (plan_of[o.item] >= 0) {
        const uint64_t h = (uint64_t)plan_of[o.item];
        add_hbm_program(ls, plans[h], hbm_blob_off[h], it.n, o.cbits_off, (uint32_t)it.ncbits,
                        d_hbm + hbm_off[h]);
      } else {
        rc = add_prog_code(ls, codes[o.item], it.conds, it.nconds, it.n, item_lb[o.item], it.seed,
                           o.cbits_off, (uint32_t)it.ncbits,
                           o.state_off == ~0ULL ? nullptr : d_states + o.state_off);
      }
      ls.items.push_back(TItem{pi, 1, 0});
    }
    acc.prepare_ms += ms_since(tp);
    mark("encode set");
    const double k0 = acc.kernel_ms;
    if (rc == DQ_OK) rc = run_launch(ls, threads, device, st, d_cbits, &acc);
    if (timing) fprintf(stderr, "[dq_run_batch] kernel         %8.3f ms\n", acc.kernel_ms - k0);
    mark("launch set");
    std::vector<HostPiece> sp, cp, hp;
    for (const Out& o : outs[c]) {
      if (rc != DQ_OK) break;
      const dq_batch_item& it = items[o.item];
      if (o.state_off != ~0ULL) sp.push_back(HostPiece{sizeof(double2) * o.state_off, it.state_out});
      cp.push_back(HostPiece{sizeof(int32_t) * o.cbits_off, it.ncbits ? it.cbits_out : nullptr});
      if (plan_of[o.item] >= 0 && it.state_out) {  // HBM item: undo its sweeps' qubit relabeling
        const uint64_t h = (uint64_t)plan_of[o.item];
        uint64_t extra = 0;
        rc = materialize_perm(d_hbm + hbm_off[h], it.n, plans[h].perm, st, &extra);
        acc.launches += (uint32_t)extra;
      }
    }
    if (c == 0)
      for (uint64_t h = 0; h < hbm_items.size(); ++h)
        hp.push_back(HostPiece{sizeof(double2) * hbm_off[h], items[hbm_items[h]].state_out});
    if (rc == DQ_OK) rc = copy_to_host(d_hbm, sizeof(double2) * hbm_amps, hp, st);
    if (rc == DQ_OK) rc = copy_to_host(d_states, sizeof(double2) * state_amps[c], sp, st);
    if (rc == DQ_OK) rc = copy_to_host(d_cbits, sizeof(int32_t) * cbit_words[c], cp, st);
    if (d_states) cudaFreeAsync(d_states, st);
    if (d_cbits) cudaFreeAsync(d_cbits, st);
    cudaStreamSynchronize(st);
    mark("outputs");
    if (rc == DQ_OK && acc.failed_inst >= 0) {
      // map (program << 40 | instruction) back to the caller's item index
      const uint64_t pi = (uint64_t)acc.failed_inst >> 40;
      const uint64_t inst = (uint64_t)acc.failed_inst & ((1ULL << 40) - 1);
      acc.failed_inst = (int64_t)((outs[c][pi].item << 40) | inst);
      rc = fail(DQ_ERR_UNSUPPORTED, "item " + std::to_string(outs[c][pi].item) + ", instruction " +
                                        std::to_string(inst) + ": unsupported generic gate");
    }
  }
  if (d_hbm) cache_free(device, sizeof(double2) * hbm_amps, d_hbm);
  acc.hbm_items = (uint32_t)hbm_items.size();
  // large states: the HBM engine, one state per size reused across items
  dq_state_t h = nullptr;
  for (uint64_t k : engine_items) {
    if (rc != DQ_OK) break;
    const dq_batch_item& it = items[k];
    if (h && h->n != it.n) {
      dq_state_destroy(h);
      h = nullptr;
    }
    if (!h) rc = dq_state_create(it.n, device, &h);
    else rc = dq_state_reset(h);
    if (rc != DQ_OK) break;
    std::vector<int32_t> cb(std::max<uint64_t>(it.ncbits, 1), -1);
    dq_run_opts o{};
    o.semantics = DQ_SEM_SHOTS;
    o.exec = DQ_EXEC_FUSED;
    dq_profile prof{};
    const auto te = std::chrono::steady_clock::now();
    rc = dq_run(h, it.prog, it.ninst, it.conds, it.nconds, it.seed, cb.data(), it.ncbits, &o, &prof);
    acc.engine_ms += ms_since(te);
    acc.boundary_draws += prof.boundary_draws;
    if (rc != DQ_OK) {
      acc.failed_inst = (int64_t)((k << 40) | (uint64_t)std::max<int64_t>(prof.failed_inst, 0));
      break;
    }
    if (it.ncbits) memcpy(it.cbits_out, cb.data(), sizeof(int32_t) * it.ncbits);
    if (it.state_out) rc = dq_state_download(h, it.state_out, 1ULL << it.n);
    acc.engine_items += 1;
  }
  if (h) dq_state_destroy(h);
  stream_give(device, st);
  mark("engine items");
  if (stats) *stats = acc;
  return rc;
}

int dq_traj_plan_create(int device, uint32_t n, const dq_inst* prog, uint64_t ninst,
                        const dq_cond* conds, uint64_t nconds, uint64_t shots, uint64_t ncbits,
                        const dq_traj_opts* opts, dq_traj_plan_t* out) {
  if (!out) return fail(DQ_ERR_INVALID_ARG, "null output plan");
  *out = nullptr;
  if (n < 1 || n > kTrajMaxQubits) return fail(DQ_ERR_INVALID_ARG, "plan: n must be in 1..16");
  if (ninst && !prog) return fail(DQ_ERR_INVALID_ARG, "null program");
  if (ncbits > kTrajMaxCbits) return fail(DQ_ERR_INVALID_ARG, "at most 1024 classical bits");
  if (shots < 1 || shots > (1ULL << 40)) return fail(DQ_ERR_INVALID_ARG, "shots must be in 1..2^40");
  for (uint64_t i = 0; i < ninst; ++i) DQ_TRY(validate_inst(prog[i], n, nconds, ncbits, conds, i));
  int threads;
  uint32_t max_span, force_lb, lb, C;
  DQ_TRY(check_opts(opts, &threads, &max_span, &force_lb));
  DQ_TRY(geometry(n, max_span, force_lb, &lb, &C));
  LaunchSet ls;
  ls.C = C;
  DQ_TRY(add_program(ls, prog, ninst, conds, nconds, n, lb, 0, 0, (uint32_t)ncbits, nullptr));
  add_shots(ls, shots);
  if (ls.enc.pool.empty()) ls.enc.pool.push_back(make_double2(0, 0));

  DeviceGuard g(device);
  dq_traj_plan_t p = new (std::nothrow) dq_traj_plan_s();
  if (!p) return fail(DQ_ERR_OOM, "host allocation failed");
  p->device = device;
  p->shots = shots;
  p->ncbits = ncbits;
  auto bail = [&](int rc) {
    delete p;
    return rc;
  };
  const size_t out_bytes = sizeof(int32_t) * (size_t)shots * ncbits;
  int rc = DQ_OK;
  auto cu = [&](cudaError_t e, const char* what) {
    if (e != cudaSuccess && rc == DQ_OK) {
      cudaGetLastError();
      rc = fail(e == cudaErrorMemoryAllocation ? DQ_ERR_OOM : DQ_ERR_CUDA,
                std::string(what) + ": " + cudaGetErrorString(e));
    }
  };
  cu(cudaStreamCreateWithFlags(&p->buf.st, cudaStreamNonBlocking), "cudaStreamCreate");
  if (rc != DQ_OK) return bail(rc);
  p->buf.own_st = true;
  cudaStream_t st = p->buf.st;
  if ((rc = upload(&p->buf.ops, ls.enc.ops, st)) != DQ_OK) return bail(rc);
  if ((rc = upload(&p->buf.pool, ls.enc.pool, st)) != DQ_OK) return bail(rc);
  if ((rc = upload(&p->buf.conds, ls.conds, st)) != DQ_OK) return bail(rc);
  if ((rc = upload(&p->buf.progs, ls.progs, st)) != DQ_OK) return bail(rc);
  if ((rc = share_or_split(ls, p->buf, p->P, device, nullptr)) != DQ_OK) return bail(rc);
  if ((rc = upload(&p->buf.items, ls.items, st)) != DQ_OK) return bail(rc);
  cu(cudaMalloc((void**)&p->buf.ctr, kCtrWords * sizeof(unsigned long long)), "cudaMalloc(counters)");
  cu(cudaMalloc((void**)&p->d_cbits, std::max<size_t>(out_bytes, 4)), "cudaMalloc(cbits)");
  cu(cudaMallocHost((void**)&p->h_cbits, std::max<size_t>(out_bytes, 4)), "cudaMallocHost(cbits)");
  cu(cudaMallocHost((void**)&p->h_seed, sizeof(uint64_t)), "cudaMallocHost(seed)");
  cu(cudaMallocHost((void**)&p->h_ctr, 2 * kCtrWords * sizeof(unsigned long long)), "cudaMallocHost(counters)");
  cu(cudaEventCreate(&p->buf.e0), "cudaEventCreate");
  cu(cudaEventCreate(&p->buf.e1), "cudaEventCreate");
  if (rc != DQ_OK) return bail(rc);
  p->h_ctr[0] = 0;
  p->h_ctr[1] = 0;
  p->h_ctr[2] = ls.items.size();
  p->h_ctr[3] = 0;
  p->h_ctr[4] = kNotFailed;
  p->h_seed[0] = 0;
  TrajParams& P = p->P;
  P.ops = p->buf.ops;
  P.pool = p->buf.pool;
  P.conds = p->buf.conds;
  P.progs = p->buf.progs;
  P.items = p->buf.items;
  P.cbits_out = p->d_cbits;
  P.queue = p->buf.ctr;
  P.boundary = p->buf.ctr + 3;
  P.failed = reinterpret_cast<long long*>(p->buf.ctr + 4);
  P.nitems = ls.items.size();
  if ((rc = config_traj(threads, C, traj_smem(ls), P.tasks ? shots : P.nitems, &p->L)) != DQ_OK) return bail(rc);
  cu(cudaStreamSynchronize(st), "cudaStreamSynchronize");
  if (rc != DQ_OK) return bail(rc);
  // capture: seed -> program table, counters reset, launch, results back
  cu(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal), "cudaStreamBeginCapture");
  if (rc != DQ_OK) return bail(rc);
  cu(cudaMemcpyAsync(&p->buf.progs[0].base_seed, p->h_seed, sizeof(uint64_t),
                     cudaMemcpyHostToDevice, st), "capture seed copy");
  cu(cudaMemcpyAsync(p->buf.ctr, p->h_ctr, kCtrWords * sizeof(unsigned long long), cudaMemcpyHostToDevice,
                     st), "capture counter reset");
  if (rc == DQ_OK) rc = reset_shared(P, shots, st);
  if (rc == DQ_OK) rc = launch_traj(p->L, P, st);
  if (out_bytes)
    cu(cudaMemcpyAsync(p->h_cbits, p->d_cbits, out_bytes, cudaMemcpyDeviceToHost, st),
       "capture cbits copy");
  cu(cudaMemcpyAsync(p->h_ctr + kCtrWords, p->buf.ctr, kCtrWords * sizeof(unsigned long long),
                     cudaMemcpyDeviceToHost, st), "capture counter copy");
  cudaGraph_t graph = nullptr;
  const cudaError_t ee = cudaStreamEndCapture(st, &graph);
  p->graph = graph;
  cu(ee, "cudaStreamEndCapture");
  if (rc == DQ_OK) cu(cudaGraphInstantiate(&p->exec, p->graph, 0), "cudaGraphInstantiate");
  if (rc != DQ_OK) return bail(rc);
  p->geom.cluster_span = C;
  p->geom.clusters = p->L.clusters;
  p->geom.threads = (uint32_t)threads;
  p->geom.local_bits = lb;
  p->geom.launches = 1;
  *out = p;
  return DQ_OK;
}

int dq_traj_plan_run(dq_traj_plan_t p, uint64_t base_seed, int32_t* cbits_out,
                     dq_traj_stats* stats) {
  if (!p || !p->exec) return fail(DQ_ERR_INVALID_ARG, "null or destroyed plan");
  const size_t out_bytes = sizeof(int32_t) * (size_t)p->shots * p->ncbits;
  if (out_bytes && !cbits_out) return fail(DQ_ERR_INVALID_ARG, "null cbits output");
  DeviceGuard g(p->device);
  cudaStream_t st = p->buf.st;
  p->h_seed[0] = base_seed;
  DQ_CUDA_TRY(cudaEventRecord(p->buf.e0, st));
  DQ_CUDA_TRY(cudaGraphLaunch(p->exec, st));
  DQ_CUDA_TRY(cudaEventRecord(p->buf.e1, st));
  DQ_CUDA_TRY(cudaStreamSynchronize(st));
  float ms = 0.f;
  DQ_CUDA_TRY(cudaEventElapsedTime(&ms, p->buf.e0, p->buf.e1));
  if (out_bytes) memcpy(cbits_out, p->h_cbits, out_bytes);
  dq_traj_stats s = p->geom;
  s.boundary_draws = p->h_ctr[kCtrWords + 3];
  const long long f = (long long)p->h_ctr[kCtrWords + 4];
  s.failed_inst = f == 0x7fffffffffffffffLL ? -1 : (f & ((1LL << 40) - 1));
  s.kernel_ms = ms;
  if (stats) *stats = s;
  if (s.failed_inst >= 0)
    return fail(DQ_ERR_UNSUPPORTED, "instruction " + std::to_string(s.failed_inst) +
                                        ": unsupported generic gate reached in a trajectory");
  return DQ_OK;
}

int dq_traj_plan_destroy(dq_traj_plan_t p) {
  if (!p) return DQ_OK;
  DeviceGuard g(p->device);
  delete p;
  return DQ_OK;
}

}  // extern "C"
