// How large a contraction's products are against the largest possible one, by
// the operands' profiles along K.
//
// Digit slices hold every element of a tensor on one fixed-point grid, so the
// error of a sum of products is relative to max|T| max|V|; an FP64 dot
// product's is relative to the products it adds.  The two are the same
// thing only where some product of every contraction is near the largest
// possible, and slab maxima do not tell: a slab's large T may all meet small
// V.  So the examination takes, for every T_x and V_yz a tuple multiplies,
//     max over E of  max_{p,q} |T[x,E,p,q]|  max_r |V[y,z,E,r]|
// (the largest product of one of its W cells) and keeps the least of them over
// all (x; y,z).  Logarithms in integers make that a product of matrices in
// (max, +) of Nv^4 steps.  A lower bound comes first, from the largest V in each
// of eight stretches of E, which is enough for data without structure; only
// where it does not reach the line are all E taken (No=20/Nv=300 with the pass
// over V: 0.93 and 2.4 ms).
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace atrip_gb300 {
namespace {

constexpr int kLogOne = 19;    // log_of: bits after the point
constexpr int kLogBias = 1023;
constexpr int kProfilePairs = 32;  // (y,z) pairs of a block

__device__ __forceinline__ unsigned long long magnitude(double x) {
  return (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
}

// log2 of a magnitude plus kLogBias: exponent and mantissa bits read as one
// number, at most 0.09 below it; sums of two stay below 2^31.
__device__ __forceinline__ int log_of(unsigned long long m) { return (int)(m >> 33); }

// The pitch of a T profile t[E][x], and its bytes.
__host__ __device__ constexpr int profile_pitch(int Nv) { return (Nv + 7) / 8 * 8; }
inline size_t profile_bytes(int Nv) { return sizeof(int) * (size_t)Nv * profile_pitch(Nv); }
constexpr int kProfileSmem = 200 << 10;  // a block's limit, with its static 2 KB
inline size_t profile_smem(int Nv) { return sizeof(int) * (size_t)Nv * (kProfilePairs + 1); }

// A warp's largest magnitude into *out.
__device__ __forceinline__ void warp_max(unsigned long long m, unsigned long long *out) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long v = __shfl_xor_sync(0xffffffffu, m, o);
    m = v > m ? v : m;
  }
  if ((threadIdx.x & 31) == 0 && m > *(volatile unsigned long long *)out) atomicMax(out, m);
}

// Block of 256 threads: the least over x and the block's pairs p0 .. of the
// largest t[E][x] + v[E][pair] over E; FULL: over all E, else over the eight
// where v is largest in a stretch.  v in shared memory, 33 to a row.  The pair
// x (Nv + 1) is (x,x), which no tuple multiplies with T_x.
template <bool FULL>
__device__ __forceinline__ void least_product(const int *t, const int *v, int Nv, int64_t p0,
                                              unsigned int *out) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, pitch = profile_pitch(Nv);
  const int64_t p = p0 + lane;
  const bool valid = p < (int64_t)Nv * Nv;
  __shared__ int top[8][kProfilePairs], at[8][kProfilePairs];
  if constexpr (!FULL) {
    const int len = (Nv + 7) / 8, e1 = min(Nv, (warp + 1) * len);
    int best = -1, where = 0;  // of an empty stretch: below any v[0]
    for (int E = warp * len; E < e1; ++E) {
      const int w = v[E * (kProfilePairs + 1) + lane];
      if (w > best) {
        best = w;
        where = E;
      }
    }
    top[warp][lane] = best;
    at[warp][lane] = where;
    __syncthreads();
  }
  unsigned int least = 0xffffffffu;
  for (int x0 = warp * 8; x0 < Nv; x0 += 64) {
    int m[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    const int4 *tx = reinterpret_cast<const int4 *>(t + x0);
#pragma unroll 4
    for (int k = 0; k < (FULL ? Nv : 8); ++k) {
      const int E = FULL ? k : at[k][lane];
      const int w = FULL ? v[E * (kProfilePairs + 1) + lane] : top[k][lane];
      const int4 a = tx[(size_t)E * (pitch / 4)], b = tx[(size_t)E * (pitch / 4) + 1];
      m[0] = __viaddmax_s32(a.x, w, m[0]);
      m[1] = __viaddmax_s32(a.y, w, m[1]);
      m[2] = __viaddmax_s32(a.z, w, m[2]);
      m[3] = __viaddmax_s32(a.w, w, m[3]);
      m[4] = __viaddmax_s32(b.x, w, m[4]);
      m[5] = __viaddmax_s32(b.y, w, m[5]);
      m[6] = __viaddmax_s32(b.z, w, m[6]);
      m[7] = __viaddmax_s32(b.w, w, m[7]);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (valid && x0 + u < Nv && p != (int64_t)(x0 + u) * (Nv + 1))
        least = min(least, (unsigned int)m[u]);
  }
  least = __reduce_min_sync(0xffffffffu, least);
  if (lane == 0) atomicMin(out, least);
}

}  // namespace
}  // namespace atrip_gb300
