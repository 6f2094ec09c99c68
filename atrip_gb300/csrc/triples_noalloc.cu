// FP64 triples loop for callers that must not allocate device memory.
//
// Who needs this: hosts whose device memory is owned by someone else -- a
// quantum-chemistry code that reserves all of HBM for its own pool allocator
// at start-up, a framework that forbids cudaMalloc/cudaFree on its worker
// threads because they synchronise the whole device, or a library running
// inside such a host.  They already hold the inputs and the outputs in their
// own buffers; atrip_gpu_run_fp64_noalloc only needs those pointers.
//
// The scratch this kernel needs (the work-queue cursor, the per-CTA W
// buffers and the partial sums of the energy reduction) lives in one
// file-scope __device__ array of fixed size, kNoallocScratchBytes.  Every
// GPU that loads this library reserves that array until the process exits.
// Calls share it: the cursor is cleared by each call, and two calls whose
// kernels overlap on the GPU (different streams, or different host threads)
// race on it -- serialise them.
//
// Operands are read straight from the caller's column-major FP64 tensors
// (the layout CTF's read_all returns), so there is no upload, no re-layout
// and no tuple table: tuples are decoded from their list position and the
// (i >= j >= k) triples are enumerated in the energy loop.  The arithmetic
// is the same as the FP64 form of atrip_gpu_run (six fused particle+hole
// contractions written into W at their index permutations, Z = W + singles,
// the get_energy_{distinct,same} terms of src/atrip/Equations.cxx:101-238).
//
// Two kernels do it.  The tensor-core one forms W as triples_fp64_tc.cu does,
// from exact products of 8-bit digit slices, but has no memory for slices: it
// cuts each K chunk of the caller's tensors into shared memory as it goes.
// The other runs on FP64 instructions.  A call cannot ask the device and wait,
// so where the first applies by its sizes both are queued: a few small kernels
// examine the operands (largest elements of the tensors and of their slabs),
// the tensor-core kernel runs if they allow exact sums, and the other one
// returns at once if that succeeded.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "atrip_gb300.h"
#include "digits.cuh"
#include "engine.cuh"
#include "kprofile.cuh"
#include "sm100.cuh"

namespace atrip_gb300 {
namespace noalloc {

constexpr size_t kScratchBytes = size_t(32) << 20;  // kNoallocScratchBytes, 32 MiB
constexpr size_t kHeaderBytes = 256;                // cursor + status
constexpr int kPartialBlocks = 128;                 // energy reduction partials
constexpr size_t kPartialBytes = sizeof(double) * 4 * kPartialBlocks;
constexpr size_t kWorkspaceOffset = kHeaderBytes + kPartialBytes;
constexpr int kThreads = 256;
constexpr int kMT = 64;
constexpr int kKC = 32;

static __device__ __align__(256) unsigned char g_scratch[kScratchBytes];

// The first bytes of the scratch, cleared by every call.
struct Header {
  unsigned long long cursor;     // FP64-instruction kernel
  unsigned long long tc_cursor;  // tensor-core kernel
  int tc_ok;                     // the operands allow exact sums
  int tc_overflow;               // a level sum left its exact range
  int tc_status;                 // a bounded wait gave up
  int e_t, e_v, e_j;             // exponents of the digit grids
  // largest magnitudes of T, of the V and of the J pair; least products of T
  // with V_pphp and J_pphp (kprofile.cuh): lower bounds, exact; the latter are
  // needed
  unsigned long long t_max, v_max[2];
  unsigned int least[2][2];
  int full;
};
static_assert(sizeof(Header) <= kHeaderBytes, "header");

struct Args {
  int No, Nv;
  const double *epsi, *epsa, *tai, *T, *Vpp, *Vh, *Vp, *Jh, *Jp;
  int64_t t_begin, t_end;
  double tai_sign;
  int use_j;
  int ijkabc;
  double *e, *ect, *energies;
  unsigned char *scratch;  // device address of g_scratch
};

// (a,b,c) of list position t: walk the lexicographic a <= b <= c list
// (src/atrip/Tuples.cxx:122-134) block by block.
__device__ void decode_tuple(int64_t t, int Nv, int &a, int &b, int &c) {
  int64_t r = t;
  for (int x = 0; x < Nv; ++x) {
    const int64_t m = Nv - x, nx = m * (m + 1) / 2 - 1;
    if (r >= nx) { r -= nx; continue; }
    for (int y = x; y < Nv; ++y) {
      const int64_t ny = (Nv - y) - (y == x ? 1 : 0);
      if (r >= ny) { r -= ny; continue; }
      a = x;
      b = y;
      c = (int)(y + r + (y == x ? 1 : 0));
      return;
    }
  }
  a = b = c = 0;
}

struct Smem {
  double As[kKC][kMT + 1];
  double Bs[kKC][64 + 1];
  double red[kThreads / 32][2];
  long long slot;
  double ta[64], tb[64], tc[64];
};

// W = sum of the six fused terms, operands read in column-major order.
template <int NC>
__device__ void build_w(const Args &g, Smem &sm, double *W, const double *Vh, const double *Vp,
                        int a, int b, int c) {
  const int64_t No = g.No, Nv = g.Nv, No2 = No * No, NvNv = Nv * Nv;
  const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
  for (int t = 0; t < 6; ++t) {
    int x, w, y, z, u, v, holeT, sp, sq, sr;
    switch (t) {
      case 0: x = a; w = b; y = b; z = c; u = a; v = c; holeT = 0; sp = 1; sq = No; sr = No2; break;
      case 1: x = a; w = c; y = c; z = b; u = a; v = b; holeT = 0; sp = 1; sq = No2; sr = No; break;
      case 2: x = c; w = a; y = a; z = b; u = b; v = c; holeT = 1; sp = No2; sq = 1; sr = No; break;
      case 3: x = c; w = b; y = b; z = a; u = a; v = c; holeT = 1; sp = No2; sq = No; sr = 1; break;
      case 4: x = b; w = a; y = a; z = c; u = b; v = c; holeT = 0; sp = No; sq = 1; sr = No2; break;
      default: x = b; w = c; y = c; z = a; u = a; v = b; holeT = 1; sp = No; sq = No2; sr = 1; break;
    }
    for (int m0 = 0; m0 < No2; m0 += kMT) {
      double acc[2][NC];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < NC; ++j) acc[i][j] = 0.0;
      for (int seg = 0; seg < 2; ++seg) {
        const int K = seg == 0 ? (int)Nv : (int)No;
        for (int k0 = 0; k0 < K; k0 += kKC) {
          // particle rows T[x,E,p,q] are read with consecutive threads on
          // E (stride Nv), hole rows Vh[p,q,L,w] on p (contiguous): the
          // nearest addresses this column-major layout offers
          for (int idx = tid; idx < kMT * kKC; idx += kThreads) {
            const int row = seg == 0 ? idx / kKC : idx % kMT;
            const int kk = seg == 0 ? idx % kKC : idx / kMT;
            const int64_t m = m0 + row, k = k0 + kk;
            double val = 0.0;
            if (m < No2 && k < K) {
              const int64_t p = m % No, q = m / No;
              val = seg == 0 ? g.T[x + k * Nv + p * NvNv + q * NvNv * No]   // T[x,E,p,q]
                             : Vh[p + q * No + k * No2 + (int64_t)w * No2 * No];  // Vh[p,q,L,w]
            }
            sm.As[kk][row] = val;
          }
          for (int idx = tid; idx < NC * 8 * kKC; idx += kThreads) {
            // V_pphp columns Vp[y,z,E,r]: consecutive threads on E (stride Nv^2)
            const int col = seg == 0 ? idx / kKC : idx % (NC * 8);
            const int kk = seg == 0 ? idx % kKC : idx / (NC * 8);
            const int64_t k = k0 + kk;
            double val = 0.0;
            if (col < No && k < K) {
              if (seg == 0)
                val = Vp[y + z * Nv + k * NvNv + (int64_t)col * NvNv * Nv];  // Vp[y,z,E,r]
              else
                val = -(holeT ? g.T[u + v * Nv + col * NvNv + k * NvNv * No]     // T[u,v,r,L]
                              : g.T[u + v * Nv + k * NvNv + col * NvNv * No]);   // T[u,v,L,r]
            }
            sm.Bs[kk][col] = val;
          }
          __syncthreads();
#pragma unroll 8
          for (int kk = 0; kk < kKC; ++kk) {
            const double a0 = sm.As[kk][ty], a1 = sm.As[kk][ty + 32];
#pragma unroll
            for (int j = 0; j < NC; ++j) {
              const double bv = sm.Bs[kk][tx + 8 * j];
              acc[0][j] = fma(a0, bv, acc[0][j]);
              acc[1][j] = fma(a1, bv, acc[1][j]);
            }
          }
          __syncthreads();
        }
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int m = m0 + ty + 32 * i;
        if (m < No2) {
          const int p = m % No, q = m / No;
#pragma unroll
          for (int j = 0; j < NC; ++j) {
            const int r = tx + 8 * j;
            if (r < No) {
              const int idx = p * sp + q * sq + r * sr;
              W[idx] = (t == 0 ? 0.0 : W[idx]) + acc[i][j];
            }
          }
        }
      }
    }
    __syncthreads();
  }
}

// Z at (i,j,k): W + t1 (x) Vpphh (src/atrip/Equations.cxx:420-422).
__device__ __forceinline__ double zval(const Args &g, const Smem &sm, const double *W, int a, int b,
                                       int c, int i, int j, int k) {
  const int64_t No = g.No, Nv = g.Nv, NvNv = Nv * Nv;
  double z = W[i + No * j + No * No * k];
  z += sm.ta[i] * g.Vpp[b + c * Nv + j * NvNv + k * NvNv * No];
  z += sm.tb[j] * g.Vpp[a + c * Nv + i * NvNv + k * NvNv * No];
  z += sm.tc[k] * g.Vpp[a + b * Nv + i * NvNv + j * NvNv * No];
  return z;
}

__device__ double energy_partial(const Args &g, const Smem &sm, const double *Tb, const double *Wz,
                                 int a, int b, int c, bool distinct, double epsabc) {
  const int No = g.No;
  double sum = 0.0;
  for (int n = threadIdx.x; n < No * No * No; n += kThreads) {
    const int i = n % No, j = (n / No) % No, k = n / (No * No);
    if (i < j || j < k) continue;
    const double facjk = j == k ? 0.5 : 1.0, facij = i == j ? 0.5 : 1.0;
    const double denominator = epsabc - ((g.epsi[i] + g.epsi[j]) + g.epsi[k]);
    double value;
    if (distinct) {
      const double U = zval(g, sm, Wz, a, b, c, i, j, k), V = zval(g, sm, Wz, a, b, c, i, k, j),
                   W = zval(g, sm, Wz, a, b, c, j, i, k), X = zval(g, sm, Wz, a, b, c, j, k, i),
                   Y = zval(g, sm, Wz, a, b, c, k, i, j), Z = zval(g, sm, Wz, a, b, c, k, j, i);
      const double A = Tb[i + No * j + No * No * k], B = Tb[i + No * k + No * No * j],
                   C = Tb[j + No * i + No * No * k], D = Tb[j + No * k + No * No * i],
                   E = Tb[k + No * i + No * No * j], F = Tb[k + No * j + No * No * i];
      const double UXY = U + (X + Y), VWZ = V + (W + Z), ADE = A + (D + E), BCF = B + (C + F);
      const double first = A * U + (B * V + (C * W + (D * X + (E * Y + F * Z))));
      value = 3.0 * first + ((UXY - 2.0 * VWZ) * ADE + (VWZ - 2.0 * UXY) * BCF);
    } else {
      const double U = zval(g, sm, Wz, a, b, c, i, j, k), V = zval(g, sm, Wz, a, b, c, j, k, i),
                   W = zval(g, sm, Wz, a, b, c, k, i, j);
      const double A = Tb[i + No * j + No * No * k], B = Tb[j + No * k + No * No * i],
                   C = Tb[k + No * i + No * No * j];
      value = 3.0 * ((A * U + B * V) + C * W) - (A + (B + C)) * (U + (V + W));
    }
    sum += (2.0 * value / denominator) * (facjk * facij);
  }
  return sum;
}

__device__ double block_sum(double v, Smem &sm, int slot) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sm.red[threadIdx.x >> 5][slot] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < kThreads / 32; ++w) r += sm.red[w][slot];
  return r;
}

template <int NC>
__global__ void __launch_bounds__(kThreads) triples_noalloc_kernel(Args g) {
  __shared__ Smem sm;
  Header *h = reinterpret_cast<Header *>(g.scratch);
  if (h->tc_ok && !h->tc_overflow && !h->tc_status) return;  // the tensor-core kernel did it
  unsigned long long *cursor = &h->cursor;
  const int64_t No3 = (int64_t)g.No * g.No * g.No;
  double *Wv = reinterpret_cast<double *>(g.scratch + kWorkspaceOffset) +
               blockIdx.x * (g.use_j ? 2 : 1) * No3;
  double *Wj = Wv + No3;
  const int64_t n = g.t_end - g.t_begin;
  for (;;) {
    if (threadIdx.x == 0) {
      const unsigned long long q = atomicAdd(cursor, 1ull);
      sm.slot = q < (unsigned long long)n ? (long long)q : -1;
    }
    __syncthreads();
    const long long slot = sm.slot;
    __syncthreads();
    if (slot < 0) break;
    const int64_t t = g.t_begin + slot;
    int a, b, c;
    decode_tuple(t, g.Nv, a, b, c);
    if (threadIdx.x < g.No) {
      const int i = threadIdx.x;
      sm.ta[i] = g.tai_sign * g.tai[a + (int64_t)i * g.Nv];
      sm.tb[i] = g.tai_sign * g.tai[b + (int64_t)i * g.Nv];
      sm.tc[i] = g.tai_sign * g.tai[c + (int64_t)i * g.Nv];
    }
    build_w<NC>(g, sm, Wv, g.Vh, g.Vp, a, b, c);
    int cls = 0;  // src/atrip/Atrip.cxx:640-642
    if (a == b) cls++;
    if (b == c) cls--;
    const double epsabc = g.epsa[a] + g.epsa[b] + g.epsa[c];
    const double e = block_sum(energy_partial(g, sm, Wv, Wv, a, b, c, cls == 0, epsabc), sm, 0);
    double ect = e;
    if (g.use_j) {
      build_w<NC>(g, sm, Wj, g.Jh, g.Jp, a, b, c);
      ect = block_sum(energy_partial(g, sm, Wj, Wv, a, b, c, cls == 0, epsabc), sm, 1);
    }
    if (threadIdx.x == 0) {
      g.e[slot] = e;
      g.ect[slot] = ect;
    }
    __syncthreads();
  }
}

// ------------------------------------------------- tensor-core kernel

namespace tc {
using namespace sm100;
constexpr int kThreads = 512;
constexpr int kS = 8;           // digit slices and levels
constexpr int kChunk = 64;      // K elements per 128-byte row
constexpr int kATile = 128 * 128;
// K contributions an accumulator may hold: then the sums of levels 0..5 are
// exact whatever the digits are, 6 K 2^14 < 2^25 - 2^22 - 2^16
// (digit_sums.cuh).  In level 6, 7 K products of at most 2^14, at least 1792
// must go into a sum that passes 2^24 and comes back, so at most 280 are added
// beyond, each rounded by at most 2: below 2^-52 of the grids' largest
// product, a quarter of what an FP64 dot product of that length may lose.
// Longer sums are drained into W in pieces.
constexpr int kMaxK = 296;
constexpr int kRangeBits = 6;  // least product against the grids' largest: triples_fp64_tc.cu

// out[s] = largest magnitude of slab s of x[s + nslab c], c < count.
__global__ void column_max(const double *__restrict__ x, int64_t nslab, int64_t count,
                           unsigned long long *__restrict__ out) {
  const int64_t s = blockIdx.x * 256ll + threadIdx.x;
  if (s >= nslab) return;
  unsigned long long m = 0;
#pragma unroll 8
  for (int64_t c = blockIdx.y; c < count; c += gridDim.y) {
    const unsigned long long b = magnitude(x[s + nslab * c]);
    m = b > m ? b : m;
  }
  atomicMax(&out[s], m);
}

// The profile of T from its columns' maxima cols[x + Nv E], and the largest.
__global__ void __launch_bounds__(256) t_profile(const unsigned long long *__restrict__ cols,
                                                 int Nv, int *__restrict__ t, Header *h) {
  const int64_t i = blockIdx.x * 256ll + threadIdx.x;
  const unsigned long long m = i < (int64_t)Nv * Nv ? cols[i] : 0;
  if (i < 4) h->least[i >> 1][i & 1] = ~0u;
  if (i < (int64_t)Nv * Nv) t[(i / Nv) * profile_pitch(Nv) + i % Nv] = log_of(m);
  warp_max(m, &h->t_max);
}

// The least product of T's profile with those of 32 slabs V[y,z,E,r] (y
// fastest) a block, and the largest element.
template <bool FULL>
__global__ void __launch_bounds__(256) v_profile(const double *__restrict__ Vp,
                                                 const int *__restrict__ t, int No, int Nv,
                                                 Header *h, int which) {
  extern __shared__ int v[];
  if (FULL && !h->full) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t p0 = (int64_t)blockIdx.x * kProfilePairs, np = (int64_t)Nv * Nv;
  unsigned long long best = 0;
  for (int E = warp; E < Nv; E += 8) {
    unsigned long long m = 0;
    if (p0 + lane < np) {
      const double *p = Vp + p0 + lane + E * np;
#pragma unroll 8
      for (int r = 0; r < No; ++r) {
        const unsigned long long b = magnitude(p[(int64_t)r * Nv * np]);
        m = b > m ? b : m;
      }
    }
    v[E * (kProfilePairs + 1) + lane] = log_of(m);
    best = m > best ? m : best;
  }
  warp_max(best, &h->v_max[which]);
  __syncthreads();
  least_product<FULL>(t, v, Nv, p0, &h->least[FULL][which]);
}

// The largest magnitude of x[0 .. n) into the header.
__global__ void __launch_bounds__(256) max_kernel(const double *__restrict__ x, int64_t n,
                                                  Header *h, int which) {
  unsigned long long m = 0;
  for (int64_t i = blockIdx.x * 256ll + threadIdx.x; i < n; i += gridDim.x * 256ll) {
    const unsigned long long b = magnitude(x[i]);
    m = b > m ? b : m;
  }
  warp_max(m, &h->v_max[which]);
}

// Smallest e with x <= 127/128 2^e; false if the exponent is out of hand.
__device__ bool grid_exponent(unsigned long long bits, int *e) {
  if (bits == 0 || bits >= 0x7ff0000000000000ull) return false;
  const double x = __longlong_as_double((long long)bits);
  int k = ilogb(x) + 1;
  if (x > ldexp(127.0 / 128.0, k)) ++k;
  *e = k;
  return k >= -200 && k <= 200;
}

// The verdict; the rules of triples_fp64_tc.cu.  From the lower bounds, then, if
// they did not do, from the exact products.
__global__ void decide(int use_j, Header *h, int full) {
  if (full && !h->full) return;
  int e_t = 0, e[2] = {0, 0};
  bool ok = grid_exponent(h->t_max, &e_t);
  for (int w = 0; w < (use_j ? 2 : 1); ++w)
    ok = ok && grid_exponent(h->v_max[w], &e[w]) &&
         ldexp((double)h->least[full][w], -kLogOne) - 2 * kLogBias >= e_t + e[w] - kRangeBits;
  h->e_t = e_t;
  h->e_v = e[0];
  h->e_j = e[1];
  h->tc_ok = ok ? 1 : 0;
  h->full = ok || full ? 0 : 1;
}

struct Tail {
  uint64_t bar;
  uint32_t tmem;
  long long slot;
  int abc[3];
  double ta[64], tb[64], tc[64];
  double red[kThreads / 32];
  int row[2][128];  // p + No q of the tile's rows, p fastest and q fastest
};

__device__ __forceinline__ double i64_to_f64(long long n) {  // |n| < 2^51
  return __longlong_as_double(0x4338000000000000ll + n) - 6755399441055744.0;
}

// Four rows of digits at a time: the loads of all of them go out first.
template <class Load>
__device__ __forceinline__ void cut_rows(unsigned char *tile, int pitch, int row0, int nrows,
                                         int e, int k0, int K, Load load) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int m0 = warp; m0 < nrows; m0 += 64) {
    double x[4][2];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int m = m0 + 16 * u, k = k0 + 2 * lane + h;
        x[u][h] = m < nrows && k < K ? load(m, k) : 0.0;
      }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int m = m0 + 16 * u;
      if (m >= nrows) break;
      const unsigned long long y0 = biased(fixed63(x[u][0], e)), y1 = biased(fixed63(x[u][1], e));
#pragma unroll
      for (int s = 0; s < kS; ++s) {
        // 128-byte rows, their 16-byte groups permuted by the row (SW128)
        const int row = row0 + m;
        *reinterpret_cast<__nv_bfloat162 *>(tile + s * pitch + row * 128 +
                                            ((lane * 4) ^ ((row & 7) << 4))) =
            __floats2bfloat162_rn(digit(y0, s), digit(y1, s));
      }
    }
  }
}

// W (+)= the three groups of one pass (V: pass 0, J: pass 1).
struct Pass {
  const double *Vh, *Vp;
  int e;
  double unit;
  double *W;
};

__device__ bool build_w(const Args &g, Header *h, Tail &t, unsigned char *At, unsigned char *Bt,
                        const Pass &ps, int a, int b, int c, uint32_t &phase, uint32_t &over) {
  const int No = g.No, No2 = No * No, P = (No + 7) / 8 * 8;
  const int64_t Nv = g.Nv, NvNv = Nv * Nv;
  const int nt = (No2 + 127) / 128, rows = ((No2 + nt - 1) / nt + 7) / 8 * 8;
  const int warp = uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  for (int grp = 0; grp < 3; ++grp)
    for (int mt = 0; mt < nt; ++mt) {
      const int m0 = mt * rows;
      for (int m = threadIdx.x; m < rows; m += kThreads) {  // read again after the last drain
        const int sl = (m0 + m) / No, f = (m0 + m) - sl * No;
        t.row[0][m] = f + No * sl;
        t.row[1][m] = sl + No * f;
      }
      __syncthreads();
      int held = 0;         // K in the accumulator
      bool first = grp == 0;  // the first piece of the first group stores W
      for (int pt = 0; pt < 4; ++pt) {
        const bool tr = pt >= 2, hole = pt & 1;
        int x, w, y, z, u, v, flip;
        if (grp == 0) {
          if (!tr) { x = a; w = b; y = b; z = c; u = a; v = c; flip = 0; }
          else     { x = b; w = a; y = a; z = c; u = b; v = c; flip = 0; }
        } else if (grp == 1) {
          if (!tr) { x = a; w = c; y = c; z = b; u = a; v = b; flip = 0; }
          else     { x = c; w = a; y = a; z = b; u = b; v = c; flip = 1; }
        } else {
          if (!tr) { x = b; w = c; y = c; z = a; u = a; v = b; flip = 1; }
          else     { x = c; w = b; y = b; z = a; u = a; v = c; flip = 1; }
        }
        const int K = hole ? No : g.Nv;
        for (int k0 = 0; k0 < K; k0 += kChunk) {
          const int kc = min(kChunk, K - k0);
          // A: rows (p,q) of this tile, p fastest (natural) or q (transposed)
          const int nrows = min(rows, No2 - m0);
          const int *row = t.row[tr];
          if (!hole) {
            const double *T = g.T + x;
            cut_rows(At, kATile, 0, nrows, h->e_t, k0, K, [&](int m, int k) {
              return T[k * Nv + row[m] * NvNv];  // T[x,E,p,q]
            });
          } else {
            const double *Vh = ps.Vh + (int64_t)w * No2 * No;
            cut_rows(At, kATile, 0, nrows, ps.e, k0, K, [&](int m, int k) {
              return Vh[row[m] + k * No2];  // Vh[p,q,L,w]
            });
          }
          // B: columns r
          if (!hole)
            cut_rows(Bt, P * 128, 0, No, ps.e, k0, K, [&](int r, int k) {
              return ps.Vp[y + z * Nv + (k + r * Nv) * NvNv];  // Vp[y,z,E,r]
            });
          else
            cut_rows(Bt, P * 128, 0, No, h->e_t, k0, K, [&](int r, int k) {
              return -g.T[u + v * Nv + (flip ? r + No * k : k + No * r) * NvNv];
            });
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          tc_fence_before();
          __syncthreads();
          if (warp == 0) {
            tc_fence_after();
            const bool leader = elect_one();
            const uint64_t ad = sdesc_sw128(smem_u32(At)), bd = sdesc_sw128(smem_u32(Bt));
            const int nkk = (kc + 15) / 16;
            uint32_t acc = held > 0 ? 1 : 0;
            for (int sa = 0; sa < kS; ++sa) {
              const int n = ((kS - sa) * P + 15) & ~15;
              const int n1 = n <= 256 ? n : ((n >> 1) + 15) & ~15;
              const uint32_t id = idesc_bf16_f32(128, 0) | ((uint32_t)(n1 >> 3) << 17);
              const uint32_t id2 = idesc_bf16_f32(128, 0) | ((uint32_t)((n - n1) >> 3) << 17);
              const uint32_t d = t.tmem + sa * P;
              if (leader)
                for (int kk = 0; kk < nkk; ++kk) {
                  const uint64_t as = ad + (uint32_t)(sa * (kATile >> 4)) + 2 * kk;
                  mma_bf16(d, as, bd + 2 * kk, id, acc);
                  if (n1 < n) mma_bf16(d + n1, as, bd + (uint32_t)(n1 * 8) + 2 * kk, id2, acc);
                  acc = 1;
                }
              __syncwarp();
              acc = 1;
            }
            if (leader) mma_commit(&t.bar);
            __syncwarp();
          }
          held += kc;
          const bool ok = mbar_wait(&t.bar, phase & 1, &h->tc_status, 1);
          ++phase;
          if (__syncthreads_or(!ok)) return false;
          // the next chunk, if the accumulator can take it
          const int next = k0 + kChunk < K ? min(kChunk, K - k0 - kChunk)
                           : pt < 3        ? min(kChunk, ((pt + 1) & 1) ? No : g.Nv)
                                           : kMaxK;
          if (held + next <= kMaxK) continue;
          // drain: level sums to exact integers, one rounding, into W
          tc_fence_after();
          const int l = (warp & 3) * 32 + lane, m = m0 + l;
          const bool valid = l < rows && m < No2;
          const int sl = m / No, f = m - sl * No;
          const int base = grp == 0 ? m : grp == 1 ? f + No2 * sl : No * f + No2 * sl;
          const int step = grp == 0 ? No2 : grp == 1 ? No : 1;
          const uint32_t tb = t.tmem + ((uint32_t)((warp & 3) * 32) << 16);
          for (int c0 = (warp >> 2) * 8; c0 < No; c0 += 32) {
            float vv[kS][8];
            __syncwarp();
#pragma unroll
            for (int L = 0; L < kS; ++L) tmem_ld8(tb + L * P + c0, vv[L]);
            tmem_wait_ld();
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              const int r = c0 + q;
              if (r >= No || !valid) continue;
              constexpr uint32_t kBits = 0x4B400000u;  // 1.5 2^23: see triples_fp64_tc.cu
              uint32_t bb[kS];
#pragma unroll
              for (int L = 1; L < kS; ++L) {
                bb[L] = __float_as_uint(vv[L][q] + 12582912.f);
                over |= bb[L] ^ 0x4B000000u;
              }
              const int n1 = (int)(bb[1] - kBits);
              const int n23 = (int)(bb[2] * 256u + bb[3] - kBits * 257u);
              const int n45 = (int)(bb[4] * 256u + bb[5] - kBits * 257u);
              const int n67 = (int)(bb[6] * 256u + bb[7] - kBits * 257u);
              const long long hi = (long long)__float2int_rn(vv[0][q]) * (1 << 24) +
                                   ((long long)n1 * 65536 + n23);
              const long long lo = (long long)n45 * 65536 + n67;
              const double val = fma(i64_to_f64(lo), 0x1p-32, i64_to_f64(hi)) * ps.unit;
              double *dst = ps.W + base + r * step;
              *dst = first ? val : *dst + val;
            }
          }
          tc_fence_before();
          __syncthreads();  // the accumulator and W are used again
          held = 0;
          first = false;
        }
      }
    }
  return true;
}

// n-th (i >= j >= k) triple, n = C(i+2,3) + C(j+1,2) + k.
__device__ __forceinline__ void triple_of(int n, int &i, int &j, int &k) {
  i = (int)cbrtf(6.f * n);
  while (i * (i + 1) * (i + 2) / 6 > n) --i;
  while ((i + 1) * (i + 2) * (i + 3) / 6 <= n) ++i;
  n -= i * (i + 1) * (i + 2) / 6;
  j = (int)((sqrtf(8.f * n + 1.f) - 1.f) * 0.5f);
  while (j * (j + 1) / 2 > n) --j;
  while ((j + 1) * (j + 2) / 2 <= n) ++j;
  k = n - j * (j + 1) / 2;
}

// This thread's part of a tuple's energy (src/atrip/Equations.cxx:101-238);
// V: the three singles blocks V[b,c,..], V[a,c,..], V[a,b,..], No x No each.
__device__ double energy_partial(const Args &g, const Tail &t, const double *V, const double *Tb,
                                 const double *Wz, bool distinct, double epsabc) {
  const int No = g.No, No2 = No * No, ntri = No * (No + 1) * (No + 2) / 6;
  auto Z = [&](int i, int j, int k) {
    double z = Wz[i + No * j + No2 * k];
    z += t.ta[i] * V[j + k * No];
    z += t.tb[j] * V[No2 + i + k * No];
    z += t.tc[k] * V[2 * No2 + i + j * No];
    return z;
  };
  auto T = [&](int i, int j, int k) { return Tb[i + No * j + No2 * k]; };
  double sum = 0.0;
  for (int n = threadIdx.x; n < ntri; n += kThreads) {
    int i, j, k;
    triple_of(n, i, j, k);
    const double facjk = j == k ? 0.5 : 1.0, facij = i == j ? 0.5 : 1.0;
    const double denominator = epsabc - ((g.epsi[i] + g.epsi[j]) + g.epsi[k]);
    double value;
    if (distinct) {
      const double U = Z(i, j, k), V2 = Z(i, k, j), W = Z(j, i, k), X = Z(j, k, i),
                   Y = Z(k, i, j), Zz = Z(k, j, i);
      const double A = T(i, j, k), B = T(i, k, j), C = T(j, i, k), D = T(j, k, i),
                   E = T(k, i, j), F = T(k, j, i);
      const double UXY = U + (X + Y), VWZ = V2 + (W + Zz), ADE = A + (D + E), BCF = B + (C + F);
      const double first = A * U + (B * V2 + (C * W + (D * X + (E * Y + F * Zz))));
      value = 3.0 * first + ((UXY - 2.0 * VWZ) * ADE + (VWZ - 2.0 * UXY) * BCF);
    } else {
      const double U = Z(i, j, k), V2 = Z(j, k, i), W = Z(k, i, j);
      const double A = T(i, j, k), B = T(j, k, i), C = T(k, i, j);
      value = 3.0 * ((A * U + B * V2) + C * W) - (A + (B + C)) * (U + (V2 + W));
    }
    sum += (2.0 * value / denominator) * (facjk * facij);
  }
  return sum;
}

// One CTA of 512 threads per SM (as many as the scratch holds W for): cut a
// chunk, multiply, in turn; W accumulates in the scratch in FP64.  Bound by
// the cut, which each tuple repeats: single doubles read from a column-major
// tensor (a 32-byte sector each) and ~60 instructions an element.
// No=24/Nv=120, 2500 tuples: 19.1 ms, 70.7 on FP64 instructions.
__global__ void __launch_bounds__(kThreads, 1) kernel(Args g) {
  extern __shared__ __align__(1024) unsigned char raw[];
  unsigned char *At = reinterpret_cast<unsigned char *>(
      (reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));
  const int No = g.No, No2 = No * No, P = (No + 7) / 8 * 8;
  unsigned char *Bt = At + kS * kATile;
  Tail &t = *reinterpret_cast<Tail *>(Bt + kS * P * 128 + 1024);
  Header *h = reinterpret_cast<Header *>(g.scratch);
  if (!h->tc_ok) return;
  const int warp = uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(&t.bar, 1);
    fence_mbar_init();
  }
  for (int i = threadIdx.x; i < (kS * kATile + kS * P * 128 + 1024) / 16; i += kThreads)
    reinterpret_cast<uint4 *>(At)[i] = make_uint4(0, 0, 0, 0);
  if (warp == 0) {
    tmem_alloc(&t.tmem, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const int64_t No3 = (int64_t)No2 * No, Nv = g.Nv;
  double *Wv = reinterpret_cast<double *>(g.scratch + kWorkspaceOffset) +
               blockIdx.x * (g.use_j ? 2 : 1) * No3;
  double *Wj = Wv + No3;
  const int64_t n = g.t_end - g.t_begin;
  const Pass pv = {g.Vh, g.Vp, h->e_v, ldexp(1.0, h->e_t + h->e_v - 14 - 24), Wv};
  const Pass pj = {g.Jh, g.Jp, h->e_j, ldexp(1.0, h->e_t + h->e_j - 14 - 24), Wj};
  uint32_t phase = 0, over = 0;
  bool alive = true;
  while (alive) {
    if (threadIdx.x == 0) {
      const unsigned long long q = atomicAdd(&h->tc_cursor, 1ull);
      t.slot = q < (unsigned long long)n ? (long long)q : -1;
      if (t.slot >= 0) decode_tuple(g.t_begin + t.slot, g.Nv, t.abc[0], t.abc[1], t.abc[2]);
    }
    __syncthreads();
    const long long slot = t.slot;
    if (slot < 0) break;
    const int a = t.abc[0], b = t.abc[1], c = t.abc[2];
    if (threadIdx.x < No) {
      const int i = threadIdx.x;
      t.ta[i] = g.tai_sign * g.tai[a + i * Nv];
      t.tb[i] = g.tai_sign * g.tai[b + i * Nv];
      t.tc[i] = g.tai_sign * g.tai[c + i * Nv];
    }
    alive = build_w(g, h, t, At, Bt, pv, a, b, c, phase, over) &&
            (!g.use_j || build_w(g, h, t, At, Bt, pj, a, b, c, phase, over));
    if (!alive) break;
    // the singles' blocks in place of the A tile
    double *V = reinterpret_cast<double *>(At);
    const int64_t pair[3] = {b + c * Nv, a + c * Nv, a + b * Nv};
    for (int i = threadIdx.x; i < 3 * No2; i += kThreads)
      V[i] = g.Vpp[pair[i / No2] + (i % No2) * Nv * Nv];
    __syncthreads();
    int cls = 0;  // src/atrip/Atrip.cxx:640-642
    if (a == b) cls++;
    if (b == c) cls--;
    const double epsabc = g.epsa[a] + g.epsa[b] + g.epsa[c];
    double e[2] = {0.0, 0.0};
    for (int pass = 0; pass < (g.use_j ? 2 : 1); ++pass) {
      double sum = energy_partial(g, t, V, pass ? Wj : Wv, Wv, cls == 0, epsabc);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (lane == 0) t.red[warp] = sum;
      __syncthreads();
      if (threadIdx.x == 0)
        for (int w = 0; w < kThreads / 32; ++w) e[pass] += t.red[w];
      __syncthreads();
    }
    if (threadIdx.x == 0) {
      g.e[slot] = e[0];
      g.ect[slot] = g.use_j ? e[1] : e[0];
    }
  }
  if (over & 0xFF800000u) atomicOr(&h->tc_overflow, 1);
  // no MMA outlives the block: after a wait that gave up (its own, or another
  // block's, reported) those of the last commit may be in flight
  if (!alive && warp == 0) mbar_drain(&t.bar, (phase - 1) & 1);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(t.tmem, 512);
}

size_t smem_bytes(int no) {
  return 1024 + kS * kATile + (size_t)kS * ((no + 7) / 8 * 8) * 128 + 1024 + sizeof(Tail);
}

// By sizes: the profile of T fits the scratch, and the range's work on FP64
// instructions (~0.8 TFLOP/s here) takes several times what examining the
// whole tensors does (~5 TB/s, the lower bounds' Nv^3 steps and a few launches).
bool sizes_ok(const Args &a) {
  const double Nv = a.Nv, No = a.No, n = (double)(a.t_end - a.t_begin);
  const double nj = a.use_j ? 2.0 : 1.0;
  const double dfma = n * nj * 12.0 * No * No * No * (No + Nv) / 0.8e12;
  const double scan = 8.0 * (Nv * Nv * No * No + nj * Nv * No * (Nv * Nv + No * No)) / 5e12 +
                      nj * Nv * Nv * Nv / 2e11 + 4e-5;
  return No >= 4 && dfma > 4.0 * scan &&
         8 * (size_t)a.Nv * a.Nv + profile_bytes(a.Nv) + 256 <= kScratchBytes - kWorkspaceOffset;
}

// Queue the examination and the kernel.
int enqueue(const Args &a, int device, cudaStream_t st) {
  const int64_t Nv = a.Nv, No = a.No, nvnv = Nv * Nv;
  int *t = reinterpret_cast<int *>(a.scratch + kWorkspaceOffset);
  auto *cols = reinterpret_cast<unsigned long long *>(a.scratch + kWorkspaceOffset +
                                                      (profile_bytes((int)Nv) + 255) / 256 * 256);
  Header *h = reinterpret_cast<Header *>(a.scratch);
  ATRIP_CUDA_TRY(cudaMemsetAsync(cols, 0, 8 * nvnv, st));
  const unsigned blocks = (unsigned)((nvnv + 255) / 256);
  const dim3 grid(blocks, (unsigned)std::min<int64_t>(No * No,
                                                      std::max<int64_t>(1, 152 * 16 / blocks)));
  column_max<<<grid, 256, 0, st>>>(a.T, nvnv, No * No, cols);
  t_profile<<<blocks, 256, 0, st>>>(cols, (int)Nv, t, h);
  ATRIP_CUDA_TRY(cudaGetLastError());
  const unsigned pairs = (unsigned)((nvnv + kProfilePairs - 1) / kProfilePairs);
  for (int full = 0; full < 2; ++full) {
    auto profile = full ? v_profile<true> : v_profile<false>;
    ATRIP_CUDA_TRY(cudaFuncSetAttribute(profile, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        kProfileSmem));
    for (int w = 0; w < (a.use_j ? 2 : 1); ++w) {
      profile<<<pairs, 256, profile_smem((int)Nv), st>>>(w ? a.Jp : a.Vp, t, (int)No, (int)Nv, h, w);
      if (!full) max_kernel<<<152 * 4, 256, 0, st>>>(w ? a.Jh : a.Vh, Nv * No * No * No, h, w);
    }
    decide<<<1, 1, 0, st>>>(a.use_j, h, full);
  }
  ATRIP_CUDA_TRY(cudaGetLastError());
  int sms = 0;
  ATRIP_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  const size_t per_cta = sizeof(double) * (a.use_j ? 2 : 1) * (size_t)No * No * No;
  const int64_t fit = (int64_t)((kScratchBytes - kWorkspaceOffset) / per_cta);
  const int64_t n = a.t_end - a.t_begin;
  const int ctas = (int)std::min<int64_t>(std::min<int64_t>(sms, fit), n);
  const size_t smem = smem_bytes((int)No);
  ATRIP_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      kSmemLimit));
  kernel<<<ctas, kThreads, smem, st>>>(a);
  ATRIP_CUDA_TRY(cudaGetLastError());
  return ATRIP_OK;
}

}  // namespace tc

__device__ __forceinline__ void neumaier(double &s, double &c, double x) {
  const double t = s + x;
  if (fabs(s) >= fabs(x))
    c += (s - t) + x;
  else
    c += (x - t) + s;
  s = t;
}

// Compensated sum of e[0..n), ect[0..n) into the caller's energies[0..1],
// with the sign of src/atrip/Atrip.cxx:1108-1111.
__global__ void noalloc_sum_stage1(Args g, int64_t n) {
  __shared__ double sh[4][kThreads];
  double *partials = reinterpret_cast<double *>(g.scratch + kHeaderBytes);
  const int64_t chunk = (n + gridDim.x - 1) / gridDim.x;
  const int64_t lo = blockIdx.x * chunk, hi = min(n, lo + chunk);
  double s0 = 0, c0 = 0, s1 = 0, c1 = 0;
  for (int64_t t = lo + threadIdx.x; t < hi; t += kThreads) {
    neumaier(s0, c0, g.e[t]);
    neumaier(s1, c1, g.ect[t]);
  }
  sh[0][threadIdx.x] = s0;
  sh[1][threadIdx.x] = c0;
  sh[2][threadIdx.x] = s1;
  sh[3][threadIdx.x] = c1;
  __syncthreads();
  if (threadIdx.x == 0) {
    double a0 = 0, b0 = 0, a1 = 0, b1 = 0;
    for (int i = 0; i < kThreads; ++i) {
      neumaier(a0, b0, sh[0][i]);
      b0 += sh[1][i];
      neumaier(a1, b1, sh[2][i]);
      b1 += sh[3][i];
    }
    partials[4 * blockIdx.x + 0] = a0;
    partials[4 * blockIdx.x + 1] = b0;
    partials[4 * blockIdx.x + 2] = a1;
    partials[4 * blockIdx.x + 3] = b1;
  }
}

__global__ void noalloc_sum_stage2(Args g) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const double *partials = reinterpret_cast<const double *>(g.scratch + kHeaderBytes);
  double s0 = 0, c0 = 0, s1 = 0, c1 = 0;
  for (int b = 0; b < kPartialBlocks; ++b) {
    neumaier(s0, c0, partials[4 * b + 0]);
    c0 += partials[4 * b + 1];
    neumaier(s1, c1, partials[4 * b + 2]);
    c1 += partials[4 * b + 3];
  }
  const double sign = g.ijkabc ? 1.0 : -1.0;
  g.energies[0] = sign * (s0 + c0);
  g.energies[1] = sign * (s1 + c1);
}

template <int NC>
int launch(const Args &a, int device, cudaStream_t st) {
  int per_sm = 0, sms = 0;
  ATRIP_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, triples_noalloc_kernel<NC>,
                                                               kThreads, 0));
  ATRIP_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  const size_t per_cta = sizeof(double) * (a.use_j ? 2 : 1) * (size_t)a.No * a.No * a.No;
  const int64_t fit = (int64_t)((kScratchBytes - kWorkspaceOffset) / per_cta);
  int64_t grid = (int64_t)sms * (per_sm > 0 ? per_sm : 1);
  if (grid > fit) grid = fit;
  const int64_t n = a.t_end - a.t_begin;
  if (grid > n) grid = n;
  if (grid < 1) grid = 1;
  triples_noalloc_kernel<NC><<<(int)grid, kThreads, 0, st>>>(a);
  ATRIP_CUDA_TRY(cudaGetLastError());
  return ATRIP_OK;
}

// Device address of g_scratch on the current device.  Looked up on every
// call (cudaGetSymbolAddress is a cheap table lookup once the module is
// loaded): an address cached across calls would go stale after a
// cudaDeviceReset or a re-created primary context, which loads the module
// again elsewhere.
unsigned char *scratch_address(int *status) {
  void *p = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&p, g_scratch);
  if (e != cudaSuccess) {
    set_error(std::string("cudaGetSymbolAddress(g_scratch): ") + cudaGetErrorString(e));
    *status = ATRIP_ERR_CUDA;
    return nullptr;
  }
  *status = ATRIP_OK;
  return static_cast<unsigned char *>(p);
}

}  // namespace noalloc
}  // namespace atrip_gb300

using namespace atrip_gb300;

extern "C" int atrip_gpu_run_fp64_noalloc(int32_t no, int32_t nv, const atrip_device_inputs *in,
                                          int64_t first_iteration, int64_t max_iterations,
                                          int32_t ijkabc, int32_t use_j, double *tuple_e,
                                          double *tuple_ect, double *energies, void *stream) {
  clear_error();
  if (!in || !tuple_e || !tuple_ect || !energies) {
    set_error("null argument");
    return ATRIP_ERR_ARGUMENT;
  }
  if (no < 1 || no > 64 || nv < 1 || nv > 1023) {
    set_error("No must be in [1, 64] and Nv in [1, 1023]");
    return ATRIP_ERR_UNSUPPORTED;
  }
  if (!in->epsi || !in->epsa || !in->tai || !in->tabij || !in->vabij || !in->vijka || !in->vabci) {
    set_error("a required input pointer is null");
    return ATRIP_ERR_ARGUMENT;
  }
  if (first_iteration < 0 || max_iterations < 0) {
    set_error("negative iteration bound");
    return ATRIP_ERR_ARGUMENT;
  }
  const size_t per_cta = sizeof(double) * 2 * (size_t)no * no * no;
  if (per_cta > noalloc::kScratchBytes - noalloc::kWorkspaceOffset) {
    set_error("No=" + std::to_string(no) + " needs " + std::to_string(per_cta) +
              " bytes of scratch per CTA; the no-allocation entry point has " +
              std::to_string(noalloc::kScratchBytes - noalloc::kWorkspaceOffset));
    return ATRIP_ERR_UNSUPPORTED;
  }
  int device = 0;
  ATRIP_CUDA_TRY(cudaGetDevice(&device));
  int status = ATRIP_OK;
  unsigned char *scratch = noalloc::scratch_address(&status);
  if (!scratch) return status;
  const int64_t n_all = atrip_gpu_n_tuples(nv);
  int64_t t_end = n_all;
  if (max_iterations != 0 && max_iterations + 1 < t_end) t_end = max_iterations + 1;
  const int64_t t_begin = first_iteration < t_end ? first_iteration : t_end;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  noalloc::Args a;
  a.No = no;
  a.Nv = nv;
  a.epsi = in->epsi;
  a.epsa = in->epsa;
  a.tai = in->tai;
  a.T = in->tabij;
  a.Vpp = in->vabij;
  a.Vh = in->vijka;
  a.Vp = in->vabci;
  a.Jh = in->jijka;
  a.Jp = in->jabci;
  a.t_begin = t_begin;
  a.t_end = t_end;
  a.tai_sign = ijkabc ? -1.0 : 1.0;
  a.use_j = (use_j && in->jijka && in->jabci) ? 1 : 0;
  a.ijkabc = ijkabc ? 1 : 0;
  a.e = tuple_e;
  a.ect = tuple_ect;
  a.energies = energies;
  a.scratch = scratch;
  // the cursor must start at zero; the partials are overwritten by every call
  ATRIP_CUDA_TRY(cudaMemsetAsync(scratch, 0, noalloc::kHeaderBytes, st));
  const int64_t n = t_end - t_begin;
  if (n > 0) {
    int rc = noalloc::tc::sizes_ok(a) ? noalloc::tc::enqueue(a, device, st) : ATRIP_OK;
    if (rc != ATRIP_OK) return rc;
    switch ((no + 7) / 8) {
      case 1: rc = noalloc::launch<1>(a, device, st); break;
      case 2: rc = noalloc::launch<2>(a, device, st); break;
      case 3: rc = noalloc::launch<3>(a, device, st); break;
      case 4: rc = noalloc::launch<4>(a, device, st); break;
      case 5: rc = noalloc::launch<5>(a, device, st); break;
      case 6: rc = noalloc::launch<6>(a, device, st); break;
      case 7: rc = noalloc::launch<7>(a, device, st); break;
      default: rc = noalloc::launch<8>(a, device, st); break;
    }
    if (rc != ATRIP_OK) return rc;
  }
  ATRIP_CUDA_TRY(cudaMemsetAsync(scratch + noalloc::kHeaderBytes, 0, noalloc::kPartialBytes, st));
  noalloc::noalloc_sum_stage1<<<n > 0 ? noalloc::kPartialBlocks : 1, noalloc::kThreads, 0, st>>>(a, n);
  ATRIP_CUDA_TRY(cudaGetLastError());
  noalloc::noalloc_sum_stage2<<<1, 32, 0, st>>>(a);
  ATRIP_CUDA_TRY(cudaGetLastError());
  return ATRIP_OK;
}
