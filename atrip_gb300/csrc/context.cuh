// Internal definition of the opaque atrip_gpu_context (shared by the
// single-system and batch entry points).
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <vector>

#include "atrip_gb300.h"
#include "engine.cuh"
#include "fp64_tc.cuh"
#include "split.cuh"

struct atrip_gpu_context {
  int No = 0, Nv = 0, device = 0, sm_count = 0;
  int field = ATRIP_FIELD_REAL;  // enum atrip_field: doubles per element = 1 + field
  int64_t n_tuples = 0;
  int n_triples = 0;
  bool have[ATRIP_N_TENSORS] = {};
  atrip_gb300::DeviceTensors dt;
  uint32_t *d_tuples = nullptr;
  uint32_t *d_triples = nullptr;
  double *d_e = nullptr, *d_ect = nullptr;
  int64_t e_lo = 0, e_hi = 0;  // tuple range holding energies of the last run
  int last_kernel = ATRIP_KERNEL_NONE;
  double last_sums[4] = {};    // (sum, compensation) of e and ect over that range
  double *d_workspace = nullptr;
  size_t workspace_doubles = 0;
  unsigned long long *d_queue = nullptr;
  double *d_partials = nullptr, *d_sum = nullptr;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  atrip_gb300::SplitState split;
  // FP64 form on the tensor cores.  Held (TcGuard) by whatever uses or frees it:
  // a call on the context or on a batch of it, or another thread that needs the
  // memory while the context is idle
  atrip_gb300::TcState tc;
  atrip_gb300::TcBuffers tcb;
  std::atomic<bool> tc_held{false};
  atrip_gb300::TcBuffers tcs;  // split forms on the same kernel
  atrip_tuning tune = {};
  // processing order of the last range (tuple_block > 1), see build_order
  std::vector<uint32_t> h_tuples;  // packed list, host copy
  uint32_t *d_order = nullptr;
  int64_t order_cap = 0, order_lo = -1, order_hi = -1;
  int order_block = 0;
};

namespace atrip_gb300 {

class TcGuard {
 public:
  explicit TcGuard(atrip_gpu_context *c);
  ~TcGuard() { c_->tc_held.store(false, std::memory_order_release); }
  TcGuard(const TcGuard &) = delete;
  TcGuard &operator=(const TcGuard &) = delete;

 private:
  atrip_gpu_context *c_;
};

// The FP64 slices are a copy the engine can do without.  free_tc drops them,
// their buffers and what is known of the operands; give_back keeps the verdict
// where the operands were found not to allow the form.  The caller holds the
// context's TcGuard.
void free_tc(atrip_gpu_context *c);
void give_back(atrip_gpu_context *c);

}  // namespace atrip_gb300
