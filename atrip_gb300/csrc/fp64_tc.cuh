// FP64 form on the tensor cores: operands cut into eight 8-bit digit slices,
// exact integer sums in FP32 accumulators, FP64 recombination and energy.
// State kept per context and the entry points used by atrip_gpu_run and the
// batch (kernel and arithmetic in triples_fp64_tc.cu).
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

#include "engine.cuh"

namespace atrip_gb300 {

struct TcState {
  void *impl = nullptr;
  bool tried = false;        // the operands were examined (and cut, if usable)
  bool usable = false;       // digit slices are ready
  bool tried_j = false, usable_j = false;  // the same for the (cT) intermediates
  uint64_t generation = 0;   // bumped whenever device buffers change
};

// Forget (and free) everything cut from the uploaded tensors.
void tc_free(TcState &s);

// Whether this form serves a system of these sizes at all.
bool tc_sizes_ok(int No, int Nv, int64_t n_tuples, bool cplx);

// The processing order of its tuples (see build_order), 0 = list order.
int tc_tuple_block(int No, int Nv, int slices, int sm_count);
constexpr int kTcFp64Slices = 8;

// Examine the operands, cut the slices and build the tensor maps, once per
// upload.  ATRIP_OK with *usable = false where the data or the free memory
// rule the form out (the caller then runs the DFMA kernel).
int tc_prepare(TcState &s, const DeviceTensors &dt, int No, int Nv, bool cplx, bool use_j,
               cudaStream_t st, int64_t *launches, bool *usable);

// The split-precision forms' slices on the same kernel: S slices of the
// operands ops[] = {T rows natural, transposed, V_hhhp natural, transposed,
// V_pphp, T_uv, T_uv^T} (pitch Kp, holes 64), unit the weight of level 0; the
// (cT) pair {J_hhhp natural, transposed, J_pphp}.  s owns none of them.
int tc_split_attach(TcState &s, int S, bool f16, int No, int Nv, int Kp, double unit,
                    void *const *ops);
int tc_split_attach_j(TcState &s, double unit_j, void *const *ops);

// One system of a launch.
struct TcSystem {
  TcState *state;
  const DeviceTensors *dt;
  int No, Nv, n_triples;
  const uint32_t *tuples, *triples;
  int64_t t_begin, t_end;
  bool use_j;
  double *e, *ect;
  const double2 *tri_ef;  // split forms: denominator part and weight of each triple
};

// Buffers of a launch, owned by a context or a batch.
struct TcBuffers {
  void *h_desc = nullptr, *d_desc = nullptr;  // descriptor table (pinned host, device)
  int64_t *h_prefix = nullptr, *d_prefix = nullptr;
  void *planes = nullptr;  // per-CTA W cells and W
  size_t planes_bytes = 0;
  // [0] bounded-wait status, [1 + k] a sum of system k left its exact range
  int *h_flags = nullptr, *d_flags = nullptr;
  unsigned long long *d_queue = nullptr;
  int cap = 0;
  // launch layout of the last tc_launch_prepare
  int n = 0, S = 8, nc = 1;
  int pieces = 1;  // items a row tile's sums are formed in
  bool split = false, f16 = false;
  int lay_no = 0, lay_cells = 0, lay_pass = 1, nslots = 0, nbslots = 0, aslot = 0,
      bslot = 0, grid = 0;
  size_t smem = 0;
  int64_t total = 0;
  // set by the owner: test of a wait that runs out, after so many SM cycles (0: off)
  long long unpublished = 0;
};
void tc_buffers_free(TcBuffers &b);

// Size the buffers for these systems and fill the host descriptor table.
// max_slots: operand ring depth limit, 0 = as many as fit.
int tc_launch_prepare(const TcSystem *sys, int n, double tai_sign, int sm_count, TcBuffers &b,
                      int max_slots = 0);
// Table copies, queue and flag reset, the launch and the flags' copy back, on
// st (capturable).
int tc_launch_enqueue(const TcBuffers &b, const uint32_t *order, cudaStream_t st,
                      int64_t *launches);
// After the launch has finished: its status.  *rerun = true where systems'
// sums left their exact range; those are barred from this form until their
// tensors are uploaded anew, and the caller runs them by the DFMA kernel.
int tc_launch_check(const TcBuffers &b, TcState *const *states, bool *rerun);

}  // namespace atrip_gb300
