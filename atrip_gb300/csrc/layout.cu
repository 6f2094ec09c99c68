// Layout transforms applied once at upload time, and the compensated energy
// reduction.
//
// atrip cuts its inputs into slices at start-up (SliceUnion::init ->
// slice_into_buffer, src/atrip/SliceUnion.cxx:305-332,
// src/atrip/Unions.hpp:77-278) and ships them between ranks per tuple.  Here
// every input is re-laid out once in HBM so that every contraction operand
// (a row of T_x, a column of V_yz, ...) is a contiguous run, and is then read
// in place for every tuple.
#include "engine.cuh"

namespace atrip_gb300 {
namespace {

// 4-D permutation as a gather: coalesced stores, strided loads.  Runs once
// per uploaded tensor.
// Box n0 x n1 x n2 x n3: dst[i . t] = src[i . s] (strides in elements).
// With t the packed strides of the box the stores are coalesced.
struct Box4 {
  int64_t n[4], s[4], t[4];
};

template <typename T>
__global__ void permute4_kernel(T *__restrict__ dst, const T *__restrict__ src, Box4 b) {
  const int64_t total = b.n[0] * b.n[1] * b.n[2] * b.n[3];
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    int64_t r = idx;
    const int64_t i0 = r % b.n[0];
    r /= b.n[0];
    const int64_t i1 = r % b.n[1];
    r /= b.n[1];
    const int64_t i2 = r % b.n[2];
    const int64_t i3 = r / b.n[2];
    dst[i0 * b.t[0] + i1 * b.t[1] + i2 * b.t[2] + i3 * b.t[3]] =
        src[i0 * b.s[0] + i1 * b.s[1] + i2 * b.s[2] + i3 * b.s[3]];
  }
}

// Neumaier accumulation of (s, c) += x.
__device__ __forceinline__ void neumaier(double &s, double &c, double x) {
  const double t = s + x;
  if (fabs(s) >= fabs(x))
    c += (s - t) + x;
  else
    c += (x - t) + s;
  s = t;
}

constexpr int kSumThreads = 256;

// (s, c) += (s2, c2): the leading parts with Neumaier's step, which leaves
// the rounding error of their sum in c.
__device__ __forceinline__ void neumaier_join(double &s, double &c, double s2, double c2) {
  neumaier(s, c, s2);
  c += c2;
}

// Sum of the 256 threads' pairs (sx, cx), (sy, cy) in a fixed tree order;
// thread 0 holds the result.
__device__ void pair_block_sum(double &sx, double &cx, double &sy, double &cy) {
  __shared__ double sh[kSumThreads / 32][4];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double a = __shfl_down_sync(0xffffffffu, sx, o), b = __shfl_down_sync(0xffffffffu, cx, o),
                 c = __shfl_down_sync(0xffffffffu, sy, o), d = __shfl_down_sync(0xffffffffu, cy, o);
    neumaier_join(sx, cx, a, b);
    neumaier_join(sy, cy, c, d);
  }
  if ((threadIdx.x & 31) == 0) {
    double *w = sh[threadIdx.x >> 5];
    w[0] = sx;
    w[1] = cx;
    w[2] = sy;
    w[3] = cy;
  }
  __syncthreads();
  if (threadIdx.x == 0)
    for (int w = 1; w < kSumThreads / 32; ++w) {
      neumaier_join(sx, cx, sh[w][0], sh[w][1]);
      neumaier_join(sy, cy, sh[w][2], sh[w][3]);
    }
}

// Deterministic compensated sum: block b reduces the contiguous chunk b of
// x and y; partials[4 b .. 4 b + 3] = (sx, cx, sy, cy).  Both stages join the
// threads' pairs in a tree: the joins are latency (one thread that joined 256
// pairs from shared memory, and one that joined 256 blocks' pairs from
// global memory, took ~0.1 ms of a 1.4 ms run).
__global__ void energy_sum_stage1(const double *__restrict__ x, const double *__restrict__ y,
                                  int64_t n, double *__restrict__ partials) {
  const int64_t chunk = (n + gridDim.x - 1) / gridDim.x;
  const int64_t lo = blockIdx.x * chunk, hi = min(n, lo + chunk);
  double sx = 0, cx = 0, sy = 0, cy = 0;
  for (int64_t t = lo + threadIdx.x; t < hi; t += kSumThreads) {
    neumaier(sx, cx, x[t]);
    neumaier(sy, cy, y[t]);
  }
  pair_block_sum(sx, cx, sy, cy);
  if (threadIdx.x == 0) {
    partials[4 * blockIdx.x + 0] = sx;
    partials[4 * blockIdx.x + 1] = cx;
    partials[4 * blockIdx.x + 2] = sy;
    partials[4 * blockIdx.x + 3] = cy;
  }
}

__global__ void energy_sum_stage2(const double *__restrict__ partials, int nb,
                                  double *__restrict__ out) {
  double sx = 0, cx = 0, sy = 0, cy = 0;
  if (threadIdx.x < nb) {
    const double *p = partials + 4 * threadIdx.x;
    sx = p[0];
    cx = p[1];
    sy = p[2];
    cy = p[3];
  }
  pair_block_sum(sx, cx, sy, cy);
  if (threadIdx.x == 0) {
    out[0] = sx + cx;
    out[1] = sy + cy;
    // the compensated pairs themselves, for exact merging across processes
    out[2] = sx;
    out[3] = cx;
    out[4] = sy;
    out[5] = cy;
  }
}

}  // namespace

cudaError_t launch_permute4_box(double *dst, const double *src, const int64_t n[4],
                                const int64_t s[4], const int64_t t[4], cudaStream_t st,
                                bool complex_elems) {
  Box4 b;
  for (int d = 0; d < 4; ++d) {
    b.n[d] = n[d];
    b.s[d] = s[d];
    b.t[d] = t[d];
  }
  const int64_t total = n[0] * n[1] * n[2] * n[3];
  if (total == 0) return cudaSuccess;
  int64_t blocks = (total + 255) / 256;
  if (blocks > 152 * 64) blocks = 152 * 64;
  if (complex_elems)
    permute4_kernel<double2><<<(int)blocks, 256, 0, st>>>(
        reinterpret_cast<double2 *>(dst), reinterpret_cast<const double2 *>(src), b);
  else
    permute4_kernel<double><<<(int)blocks, 256, 0, st>>>(dst, src, b);
  return cudaGetLastError();
}

cudaError_t launch_permute4(double *dst, const double *src, const int64_t n[4], const int64_t s[4],
                            cudaStream_t st, bool complex_elems) {
  const int64_t t[4] = {1, n[0], n[0] * n[1], n[0] * n[1] * n[2]};
  return launch_permute4_box(dst, src, n, s, t, st, complex_elems);
}

cudaError_t launch_energy_sum(const double *x, const double *y, int64_t n, double *partials,
                              double *out, cudaStream_t st) {
  energy_sum_stage1<<<kSumBlocks, kSumThreads, 0, st>>>(x, y, n, partials);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  static_assert(kSumBlocks <= kSumThreads, "one block pair per thread");
  energy_sum_stage2<<<1, kSumThreads, 0, st>>>(partials, kSumBlocks, out);
  return cudaGetLastError();
}

}  // namespace atrip_gb300
