// dq_handle.cuh — the state handle behind dq_state_t and the helpers the
// extern "C" translation units (dq_api.cu, dq_adjoint.cu) share.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "dq_common.cuh"
#include "dq_engine.cuh"
#include "dq_fused.cuh"
#include "dq_gates.hpp"

struct dq_state_s {
  int device = 0;
  uint32_t n = 0;
  uint64_t len = 0;
  size_t bytes = 0;
  double2* amp = nullptr;
  cudaStream_t stream = nullptr;
  dq::Scratch sc;
  dq::FusedWork fw;
  // perm[l] = physical bit position holding logical qubit l (fused runs
  // relabel swap gates instead of moving data)
  uint32_t perm[64];
  bool permuted = false;
  // >= 0: the state is the physical basis vector |lazy_basis> but memory has
  // not been written yet; the next fused sweep synthesises its input tiles
  // from it (no read of the state, no reset pass), anything else writes it
  // first (materialize_basis)
  int64_t lazy_basis = -1;
  // query buffers (marginals, CDF, sampled indices): kept and grown as needed
  // so that a query allocates nothing per call
  void* q_dev = nullptr;
  size_t q_dev_cap = 0;
  void* q_host = nullptr;  // pinned
  size_t q_host_cap = 0;
};

namespace dq {

constexpr uint32_t kMaxQubits = 34;

struct DeviceGuard {
  int prev = -1;
  explicit DeviceGuard(int dev) {
    cudaGetDevice(&prev);
    if (prev != dev) cudaSetDevice(dev);
  }
  ~DeviceGuard() {
    int cur = -1;
    cudaGetDevice(&cur);
    if (prev >= 0 && cur != prev) cudaSetDevice(prev);
  }
};

// Device buffers of state size are recycled through a per-(device, size) cache.
int cache_alloc(int device, size_t bytes, void** out);
void cache_free(int device, size_t bytes, void* p);
// Lets a kernel's launches on the current device use `bytes` of dynamic shared
// memory.  The limit belongs to the kernel and is only ever raised: launches of
// other threads and handles with other sizes share it.
int allow_shared(const void* kernel, size_t bytes);
// Whether the thread's limit (dq_debug_alloc_limit) refuses an allocation.
bool alloc_refused(size_t bytes);
// Device memory a call may try to allocate before it asks how much is free (a
// sixteenth of the device's memory): cudaMemGetInfo takes 0.4 to 4 ms next to
// live memory pools.  A call whose allocation fails asks after all.
uint64_t unasked_budget(int device);
// Non-blocking streams for calls without a handle of their own, kept for the
// next call (at most 8 per device; creating and destroying one takes 150 us).
// A stream given back has no work pending.
int stream_take(int device, cudaStream_t* out);
void stream_give(int device, cudaStream_t st);
// Pinned host staging buffers (at least `bytes`), recycled by size class.
int pinned_alloc(size_t bytes, void** out);
void pinned_free(size_t bytes, void* p);

// One device range copied to host memory: piece i covers the bytes from
// pieces[i].off to the next piece's off (the last one to `bytes`), ascending
// from 0; a null dst is skipped.  Enqueued after the work on st; complete on return.
struct HostPiece {
  size_t off;
  void* dst;
};
int copy_to_host(const void* src, size_t bytes, const std::vector<HostPiece>& pieces, cudaStream_t st);

int check_handle(dq_state_t h);            // validates and materialises a lazy basis state
int check_handle_lazy(dq_state_t h);       // validates only
int materialize_basis(dq_state_t h);
int sync_stream(dq_state_t h);
// Make the physical layout canonical (undo a pending qubit relabeling).
int canonicalize(dq_state_t h);
// Mark the layout canonical without moving data (the state is rewritten).
void reset_perm(dq_state_t h);
// Copy `count` device doubles to `out` through the handle's pinned buffer.
int read_scalars(dq_state_t h, const double* d_src, int count, double* out);
// Grow the handle's query buffers to at least dev_bytes (device) and
// host_bytes (pinned host); the stream is drained before a buffer is replaced.
int ensure_query_buffers(dq_state_t h, size_t dev_bytes, size_t host_bytes);
// Runs a program of dq_run on a small state in one launch (exact per-gate
// arithmetic; the state canonical or a pending basis state; no profile, at
// most kSmallQubits qubits and kSmallCbits classical bits).
constexpr uint32_t kSmallQubits = 12;
constexpr uint64_t kSmallCbits = 1024;
int small_run(dq_state_t h, const dq_inst* prog, uint64_t ninst, const dq_cond* conds, uint64_t nconds,
              uint64_t seed, int32_t* cbits, uint64_t ncbits, int semantics, dq_profile* prof);
int gate_qubit_count(int kind);
int validate_inst(const dq_inst& in, uint32_t n, uint64_t nconds, uint64_t ncbits,
                  const dq_cond* conds, uint64_t idx);
// Reduce a gate instruction to its kernel class (false: no matrix).
bool inst_to_op(const dq_inst& in, GateOp& op);

}  // namespace dq
