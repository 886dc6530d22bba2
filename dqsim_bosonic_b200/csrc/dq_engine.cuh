// dq_engine.cuh — host launchers of the exact per-gate kernels and the
// reduction / sampling kernels (dq_engine.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "dq_common.cuh"
#include "dq_gates.hpp"

namespace dq {

struct Scratch {            // per-handle device/pinned scratch
  double* d_partial = nullptr;   // kPartials doubles
  unsigned* d_counter = nullptr; // last-block counters
  double* h_pinned = nullptr;    // 64 doubles pinned
  unsigned long long* d_ull = nullptr;
};

constexpr int kPartials = 4096;
constexpr int kRedThreads = 512;

// One classified gate on a state of n qubits.  Returns DQ_OK or an error.
int launch_gate(double2* s, uint32_t n, const GateOp& op, cudaStream_t st, int device,
                uint64_t* launches);

// Number of per-block partial sums the p1 reduction of an n-qubit state uses.
unsigned p1_reduction_blocks(uint32_t n, int device);
// Grid of a reduction kernel over `items` work items (at most kPartials / 4 blocks).
unsigned reduction_blocks(uint64_t items, int device);
// p1 = sum over amplitudes with bit q set (device value in *d_out).
int launch_p1(const double2* s, uint32_t n, uint32_t q, Scratch& sc, double* d_out,
              cudaStream_t st, int device);
// Zero the other half, divide the kept half by norm.
int launch_collapse(double2* s, uint32_t n, uint32_t q, int outcome, double norm,
                    cudaStream_t st, int device);
int launch_set_basis(double2* s, uint32_t n, uint64_t index, cudaStream_t st, int device);

// Device doubles of workspace a marginal over these (physical) qubits needs.
uint64_t marginal_workspace(uint32_t n, const uint32_t* qubits, uint32_t k, int device);
// marginal probabilities into a device buffer d_out[2^k]; d_work holds
// marginal_workspace() doubles (nullptr: a stream-ordered temporary is used).
int launch_marginal(const double2* s, uint32_t n, const uint32_t* qubits, uint32_t k,
                    double* d_out, double* d_work, Scratch& sc, cudaStream_t st, int device);
// Consecutive gates applied in one pass (k_group).  group_add takes a gate if it
// fits the group (at most four target qubits); a group that is not worth a
// pass is launched gate by gate instead.
constexpr int kGroupOps = 12;
struct GateGroup {
  struct Op {
    GateClass cls;
    uint32_t t0, t1;      // targets (GC_DIAG: its qubits, 64: none)
    uint64_t ctrl;        // GC_PHASE: with the target
    uint32_t mat;
  };
  std::vector<Op> ops;
  std::vector<hc> mats;
  uint64_t regs = 0;
  double saved = 0.0;     // single launches less the gates' share of a pass (gate_costs)
  void clear() {
    ops.clear();
    mats.clear();
    regs = 0;
    saved = 0.0;
  }
};
bool group_add(GateGroup& g, const GateOp& op);
bool group_worth(const GateGroup& g, uint32_t n);
int launch_group(double2* s, uint32_t n, const GateGroup& g, cudaStream_t st, uint64_t* launches);
// Marginal, CDF and samples in one launch, where the distribution fits one
// block's scan and every output is summed by one thread: d_out holds the
// shots' indices, then at entry (shots + 1) / 2 * 2 the 64-bit boundary count.
bool sample_small_ok(uint32_t n, const uint32_t* qubits, uint32_t k, uint64_t shots, int device);
int launch_sample_small(const double2* s, uint32_t n, const uint32_t* qubits, uint32_t k, const uint32_t key[8],
                        uint64_t shots, uint32_t* d_out, cudaStream_t st, int device);
// Device doubles of workspace launch_cdf needs for len entries.
uint64_t cdf_workspace(uint64_t len);
// in-place inclusive prefix sum of d[len] (deterministic order), last = 1.0;
// d_work holds cdf_workspace(len) doubles (nullptr: a stream-ordered temporary).
int launch_cdf(double* d, uint64_t len, double* d_work, cudaStream_t st, int device);
// per-shot lower_bound in the CDF with device ChaCha8 draws.
int launch_sample(const double* cdf, uint64_t len, const uint32_t key[8], uint64_t shots,
                  uint32_t* d_idx, unsigned long long* d_boundary, cudaStream_t st, int device);

// sum conj(a)*b -> d_out[0..1]; sum |a|^2 -> d_out[0]
int launch_inner(const double2* a, const double2* b, uint32_t n, Scratch& sc, double* d_out,
                 cudaStream_t st, int device);
int launch_norm(const double2* a, uint32_t n, Scratch& sc, double* d_out, cudaStream_t st,
                int device);

}  // namespace dq
