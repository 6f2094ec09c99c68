// The triples kernel on the tensor cores: the FP64 form (real and complex),
// and the split forms' slices on the same structure.
//
// FP64 arithmetic on this part runs at ~1.25 TFLOP/s whichever instruction
// does it, BF16 MMAs at ~1900.  So the contractions are done as the Ozaki
// scheme does them (Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59,
// 2012): an FP64 operand is cut into integer digit slices, the slices are
// multiplied exactly by the matrix units, and the products are added up in
// wide integers and FP64.  With e the exponent above the tensor's largest
// element,
//     x = 2^(e-7) sum_{s<8} q_s 2^(-8s),   q_s integer, |q_s| <= 128,
// holds x to 2^(e-64).  Every q_s is exact in BF16, q q' is below 2^14, and
// a sum of products is exact in the FP32 accumulator while it stays below
// 2^24.  Products are grouped by level L = s + s'; levels 0..7 are kept (36
// of the 64 slice products).  What is dropped lies 2^-58 below a typical
// element of W, where the DFMA kernel's own rounding is at 2^-51.
//
// When that holds is examined, not assumed (tc_prepare and the kernel's
// overflow flag): operands must be finite; the largest product |T V| of every
// T_x with every V_yz must lie within 2^kRangeBits of the grids' largest
// (kprofile.cuh): what is lost of K products (levels 8 and up, the bits below
// the grids), at most 9 K 2^-64 of the grids' largest, is then below a third of
// K 2^-53 of that product, the bound of an FP64 dot product's error; the sums
// of levels 0..6 are exact by the rows' digit norms and where they end
// (digit_sums.cuh), in one accumulator or, for longer K, the natural and the
// transposed half in one each (level 6 may be rounded a little where the least
// product is within 2^kLooseBits); level 7's weigh 2^-70 of the grids' largest
// product, and what roundings could do to them (8 K of at most 16) stays below
// K 2^-62 of it.  Whatever fails this is run by the DFMA kernel instead.
//
// Contraction structure: the six fused particle+hole terms of
// src/atrip/Equations.cxx:455-728 pair up by their column index into three
// K-concatenated GEMMs (the partner's rows read from a transposed copy)
//   G0  rows (i,j), column k:  T_a V_bc - Vh_b T_ac + T_b V_ac - Vh_a T_bc
//   G1  rows (i,k), column j:  T_a V_cb - Vh_c T_ab + T_c V_ab - Vh_a T_bc
//   G2  rows (j,k), column i:  T_b V_ca - Vh_c T_ab + T_c V_ba - Vh_b T_ac
// An item is 128 rows of one group.  A operand: one slice of those rows per
// ring slot; B operand: the 8 slices of the columns stacked in shared memory
// (slice s at rows s P, P = columns rounded up to 8), loaded once per K
// chunk.  Slice sa of A times slices 0..7-sa of B is one MMA (two above
// N = 256) whose result columns are the level accumulators sa..7, which lie
// side by side in TMEM: no product is padded but for P.
//
// Kernel roles (512 threads, one persistent CTA per SM):
//   warp 0            TMA producer, owner of the tuple queue
//   warp 1            TMEM owner and single-thread tcgen05.mma issuer
//   warps 4..7        epilogue: level accumulators to exact integers, stored
//                     as the group's W cells
//   warps 2, 3, 8..15 energy: W in FP64, Zijk, get_energy_{distinct,same}
//                     (src/atrip/Equations.cxx:101-238), one tuple behind
//
// What bounds it: the MMA issuer where there are few columns (an MMA of N <=
// 96 costs ~50 cycles, its issue and its share of a slot's wait and signal as
// much), shared memory beyond (an MMA of N columns reads 4 KB of A and 32 N
// bytes of B at ~118 B per cycle, and the TMA's writes take their part), the
// operand stream from L2 and HBM (No=24/Nv=240: 47 B per cycle and SM) and, at
// large No, the energy warps' gathers.  Whole runs against the DFMA kernel:
// No=24/Nv=240, 8000 tuples, 316 -> 10.4 ms (1.11 -> 34 TFLOP/s
// FP64-equivalent); No=37/Nv=151 with (cT), 900 tuples, 229.6 -> 7.7 ms;
// No=8/Nv=40, the whole list, 6.2 -> 0.92 ms; complex No=13/Nv=50, 9000
// tuples, 90.8 -> 3.7 ms.  Error of the tuple energies against quad precision,
// 2-norm, No = 8..37: 0.9 to 1.1e-16 and 1.8 to 2.7e-16 for (cT), DFMA kernel
// 0.8 to 1.1e-16 and 4.2 to 6.2e-16.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <type_traits>

#include "complex.cuh"
#include "digit_sums.cuh"
#include "digits.cuh"
#include "engine.cuh"
#include "fp64_tc.cuh"
#include "kprofile.cuh"
#include "recip.cuh"
#include "sm100.cuh"

namespace atrip_gb300 {
namespace {

using namespace sm100;

constexpr int kThreads = 512;
constexpr int kS = 8;                       // digit slices and levels of the FP64 form
constexpr int kKChunk = 64;                 // BF16 elements per 128-byte row
constexpr int kMaxSlots = 10;               // A ring
constexpr int kTupleSlots = 4;
constexpr int kEnergyWarps = 10;
constexpr int kEnergyThreads = kEnergyWarps * 32;
constexpr int kT1 = 64;  // doubles per t1 row: No <= 64, or No <= 32 complex
constexpr int kTailBytes = 576 + 3 * kT1 * 8 + 16 * 8;
constexpr int kRangeBits = 6;               // least product against 2^(eT+eV)
constexpr int kLooseBits = 4;               // the same, for loose level sums
constexpr int kBlocksZ = 3;                 // column blocks stored for a complex operand

enum : int { kErrFull = 1, kErrEmpty = 2, kErrAccFull = 3, kErrAccEmpty = 4 };

// A operands by row order (natural, transposed) and component ([1]: imaginary
// parts of a complex system); B operands.
struct TcMaps {
  CUtensorMap Ta[2][2], Vh[2][2], Vp, TpN, TpT;
  CUtensorMap Jh[2][2], Jp;  // (cT) intermediates in place of V_hhhp, V_pphp
};
constexpr int kMapsMain = 11, kMaps = 16;
static_assert(sizeof(TcMaps) == kMaps * sizeof(CUtensorMap), "maps are contiguous");

struct TcDesc {
  TcMaps maps;
  const double *epsi, *epsa, *tai, *Vhh;
  const uint32_t *tuples, *triples;
  const double2 *tri_ef;
  double *e, *ect;
  double unit, unit_j;  // weight of a W cell's high part
  double tai_sign;
  int64_t t_begin;
  int No, Nv, P, rows, spp, n_triples, use_j;
};

struct TcArgs {
  const TcDesc *sys;
  const int64_t *prefix;
  int nsys;
  int64_t total;
  int claim;              // tuples taken from the queue at once, <= 32
  const uint32_t *order;  // processing order of a single system's range
  unsigned long long *queue;
  int *flags;
  void *planes;       // [CTA][parity][pass][group][cell]
  double *wd;         // [CTA][pass][cell]
  int lay_cells, lay_pass, nslots, nbslots, aslot, bslot;
  // test of a wait that runs out: no tuple is published, and the producer waits
  // for one this many SM cycles (0: off).  A limit that every wait takes from
  // here costs the issuer 1 %
  long long unpublished;
};

__device__ __forceinline__ void bar_sync(int id, int n) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}
__device__ __forceinline__ bool bar_and(int id, int n, bool v) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "bar.red.and.pred q, %2, %3, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)v), "r"(id), "r"(n)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ void tensormap_acquire(const void *map) {
  asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(
                   reinterpret_cast<uint64_t>(map))
               : "memory");
}

// |n| < 2^51: 1.5 2^52 + n holds n in its low mantissa bits.
__device__ __forceinline__ double i64_to_f64(long long n) {
  return __longlong_as_double(0x4338000000000000ll + n) - 6755399441055744.0;
}

// Operand sources of group g, part pt of tuple (a,b,c): natural, then
// transposed rows; in each the particle, then the hole contraction; for a
// complex system in each of those A's real, then its imaginary parts.
// A complex product is four real ones: columns [re | im] of
//   A_re [V_re | V_im] + A_im [-V_im | V_re]              (particle)
//   A_re [-T_re | -T_im] + A_im [-T_im | T_re]            (hole, conj(V_hhhp))
// whose column blocks are neighbours in planes (-im, re, im) of V and
// (-re, -im, re) of T: blk is the first one.
template <bool CPLX>
struct TcParts {
  static constexpr int kCount = CPLX ? 8 : 4;
  __device__ static __forceinline__ bool hole(int pt) { return (CPLX ? pt >> 1 : pt) & 1; }
};
struct TcPart {
  const CUtensorMap *amap, *bmap;
  int ax, by, bz, blk;
};
template <bool CPLX>
__device__ __forceinline__ TcPart part_of(const TcMaps &m, int g, int pt, int a, int b, int c,
                                          int pass) {
  int x, w, y, z, u, v, flip;
  const bool tr = pt >= TcParts<CPLX>::kCount / 2;
  const int im = CPLX ? pt & 1 : 0;
  if (g == 0) {
    if (!tr) { x = a; w = b; y = b; z = c; u = a; v = c; flip = 0; }
    else     { x = b; w = a; y = a; z = c; u = b; v = c; flip = 0; }
  } else if (g == 1) {
    if (!tr) { x = a; w = c; y = c; z = b; u = a; v = b; flip = 0; }
    else     { x = c; w = a; y = a; z = b; u = b; v = c; flip = 1; }
  } else {
    if (!tr) { x = b; w = c; y = c; z = a; u = a; v = b; flip = 1; }
    else     { x = c; w = b; y = b; z = a; u = a; v = c; flip = 1; }
  }
  TcPart p;
  if (!TcParts<CPLX>::hole(pt)) {
    p.amap = &m.Ta[im][tr];
    p.ax = x;
    p.bmap = pass ? &m.Jp : &m.Vp;
    p.bz = z;
    p.by = y;
    p.blk = im ? 0 : 1;
  } else {
    p.amap = pass ? &m.Jh[im][tr] : &m.Vh[im][tr];
    p.ax = w;
    p.bmap = flip ? &m.TpT : &m.TpN;
    p.bz = v;
    p.by = u;
    p.blk = im ? 1 : 0;
  }
  return p;
}

// What a kernel instantiation multiplies: S digit slices and levels; CPLX a
// complex system; PIECES the items a row tile's sums are formed in, 2: its
// natural and its transposed half, where K is too long for exact sums in one
// (a constant: the issuer pays for every instruction; a run-time choice took
// No=8/Nv=40 from 0.91 to 0.93 .. 0.97 ms); SPLIT the split-precision forms'
// slices, BF16 of radix 2^8 or (F16) FP16 of radix 2^11, and their energy
// arithmetic.
template <int S_, bool CPLX_, bool SPLIT_, bool F16_, int PIECES_ = 1>
struct Fmt {
  static constexpr int S = S_;
  static constexpr bool CPLX = CPLX_;
  static constexpr int PIECES = PIECES_;
  static constexpr bool SPLIT = SPLIT_;  // an A ring slot holds all slices of a chunk
  __device__ static constexpr int radix() { return F16_ ? 2048 : 256; }
  // A level sum of the split forms as an integer.  FP16 digits: level 1 adds up
  // two products of at most 2^20 for each of up to 2047 K, which 32 bits do not
  // hold from K = 1024 on; every other one stays below 2^31.  It is taken apart
  // as 2048 a + b by adding 1.5 2^23, which leaves an integer below 2^22 in the
  // low mantissa bits (the conversion to 64 bits: No=53/Nv=201 11.4 -> 13.0 ms).
  __device__ static __forceinline__ long long level(int L, float v) {
    if (!F16_ || L == 0) return __float2int_rn(v);
    const float a = fmaf(v, 1.f / 2048.f, 12582912.f), b = fmaf(a - 12582912.f, -2048.f, v);
    return (long long)((int)__float_as_uint(a) - 0x4B400000) * 2048 +
           ((int)__float_as_uint(b + 12582912.f) - 0x4B400000);
  }
  __device__ static constexpr uint32_t idesc(int n) {
    return F16_ ? idesc_f16_f32(128, n) : idesc_bf16_f32(128, n);
  }
};
template <int PIECES>
using FmtFp64 = Fmt<kS, false, false, false, PIECES>;
template <int PIECES>
using FmtZ = Fmt<kS, true, false, false, PIECES>;

struct TcSlot {
  int64_t t;  // list position, -1 = no more work
  int a, b, c, s;
};

struct TcSinglesCtx {
  const double *Vbc, *Vac, *Vab;
  const double *ta, *tb, *tc;
};

__device__ __forceinline__ double zval(const double *W, const TcSinglesCtx &s, int No, int i, int j,
                                       int k) {
  double z = W[i + No * j + No * No * k];
  z += s.ta[i] * s.Vbc[j + k * No];
  z += s.tb[j] * s.Vac[i + k * No];
  z += s.tc[k] * s.Vab[i + j * No];
  return z;
}

// This thread's part of a tuple's energy, T from Tb and Z from Wz + singles:
// the expressions of the DFMA kernel's energy loop, with its division.
// SPLIT: the split forms' arithmetic, the occupied part of the denominator
// and the weight from a table and a refined reciprocal for the division.
template <bool SPLIT>
__device__ __forceinline__ double energy_partial(const TcDesc &d, const double *Tb,
                                                 const double *Wz, const TcSinglesCtx &s,
                                                 bool distinct, double epsabc, int er) {
  const int No = d.No;
  double sum = 0.0;
  for (int n = er; n < d.n_triples; n += kEnergyThreads) {
    const uint32_t pk = d.triples[n];
    const int i = pk & 0xff, j = (pk >> 8) & 0xff, k = (pk >> 16) & 0xff;
    const double2 ef = SPLIT ? d.tri_ef[n] : make_double2(0.0, 0.0);
    const double fac = SPLIT ? ef.y : (j == k ? 0.5 : 1.0) * (i == j ? 0.5 : 1.0);
    const double denominator =
        epsabc - (SPLIT ? ef.x : (d.epsi[i] + d.epsi[j]) + d.epsi[k]);
    double value;
    if (distinct) {
      const double U = zval(Wz, s, No, i, j, k), V = zval(Wz, s, No, i, k, j),
                   W = zval(Wz, s, No, j, i, k), X = zval(Wz, s, No, j, k, i),
                   Y = zval(Wz, s, No, k, i, j), Z = zval(Wz, s, No, k, j, i);
      const double A = Tb[i + No * j + No * No * k], B = Tb[i + No * k + No * No * j],
                   C = Tb[j + No * i + No * No * k], D = Tb[j + No * k + No * No * i],
                   E = Tb[k + No * i + No * No * j], F = Tb[k + No * j + No * No * i];
      const double UXY = U + (X + Y), VWZ = V + (W + Z), ADE = A + (D + E), BCF = B + (C + F);
      const double first = A * U + (B * V + (C * W + (D * X + (E * Y + F * Z))));
      value = 3.0 * first + ((UXY - 2.0 * VWZ) * ADE + (VWZ - 2.0 * UXY) * BCF);
    } else {
      const double U = zval(Wz, s, No, i, j, k), V = zval(Wz, s, No, j, k, i),
                   W = zval(Wz, s, No, k, i, j);
      const double A = Tb[i + No * j + No * No * k], B = Tb[j + No * k + No * No * i],
                   C = Tb[k + No * i + No * No * j];
      value = 3.0 * ((A * U + B * V) + C * W) - (A + (B + C)) * (U + (V + W));
    }
    if constexpr (SPLIT)
      sum = fma(value, recip_nr(denominator) * fac, sum);
    else
      sum += (2.0 * value / denominator) * fac;
  }
  return sum;
}

// The same for a complex system: the expressions of the complex DFMA kernel.
// W as planes of real and imaginary parts, cells apart.
struct TcSinglesZ {
  const double2 *Vbc, *Vac, *Vab, *ta, *tb, *tc;
};
__device__ __forceinline__ double2 zval_z(const double *W, size_t cells, const TcSinglesZ &s, int No,
                                          int i, int j, int k) {
  const int x = i + No * j + No * No * k;
  double2 z = make_double2(W[x], W[cells + x]);
  z = cadd(z, cmul(s.ta[i], s.Vbc[j + k * No]));
  z = cadd(z, cmul(s.tb[j], s.Vac[i + k * No]));
  z = cadd(z, cmul(s.tc[k], s.Vab[i + j * No]));
  return z;
}
__device__ __forceinline__ double energy_partial_z(const TcDesc &d, const double *Tb,
                                                   const double *Wz, size_t cells,
                                                   const TcSinglesZ &s, bool distinct,
                                                   double epsabc, int er) {
  const int No = d.No;
  const double2 *epsi = reinterpret_cast<const double2 *>(d.epsi);
  double sum = 0.0;
  for (int n = er; n < d.n_triples; n += kEnergyThreads) {
    const uint32_t pk = d.triples[n];
    const int i = pk & 0xff, j = (pk >> 8) & 0xff, k = (pk >> 16) & 0xff;
    const double fac = (j == k ? 0.5 : 1.0) * (i == j ? 0.5 : 1.0);
    const double2 eijk = cadd(cadd(epsi[i], epsi[j]), epsi[k]);
    const double2 den = make_double2(epsabc - eijk.x, -eijk.y);
    auto T = [&](int p, int q, int r) {
      const int x = p + No * q + No * No * r;
      return make_double2(Tb[x], -Tb[cells + x]);  // conj(T)
    };
    auto Z = [&](int p, int q, int r) { return zval_z(Wz, cells, s, No, p, q, r); };
    double2 value;
    if (distinct) {
      // one permutation after the other: sums over the even (ijk, jki, kij)
      // and the odd ones, and the products
      double2 first = make_double2(0.0, 0.0), zs[2], ts[2];
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        const int p = i, q = o ? k : j, r = o ? j : k;
        const double2 z0 = Z(p, q, r), z1 = Z(q, r, p), z2 = Z(r, p, q);
        const double2 t0 = T(p, q, r), t1 = T(q, r, p), t2 = T(r, p, q);
        first = cadd(first, cadd(cmul(t0, z0), cadd(cmul(t1, z1), cmul(t2, z2))));
        zs[o] = cadd(z0, cadd(z1, z2));
        ts[o] = cadd(t0, cadd(t1, t2));
      }
      const double2 second = cmul(csub(zs[0], cscale(2.0, zs[1])), ts[0]);
      const double2 third = cmul(csub(zs[1], cscale(2.0, zs[0])), ts[1]);
      value = cadd(cscale(3.0, first), cadd(second, third));
    } else {
      const double2 U = Z(i, j, k), V = Z(j, k, i), W = Z(k, i, j);
      const double2 A = T(i, j, k), B = T(j, k, i), C = T(k, i, j);
      value = csub(cscale(3.0, cadd(cadd(cmul(A, U), cmul(B, V)), cmul(C, W))),
                   cmul(cadd(A, cadd(B, C)), cadd(U, cadd(V, W))));
    }
    sum += cdiv_re(cscale(2.0, value), den) * fac;
  }
  return sum;
}


// The MMA issuer's state, carried from tuple to tuple.
struct MmaRole {
  int st, bs;              // A and B ring slots of the next operands
  uint32_t ph, item;       // the A slot's phase; items so far
  int nslots, nbslots, aslot, bslot;
  uint32_t ring_a, ring_b, tm;
  uint64_t *afull, *aempty, *accf, *acce;
  bool leader;
  int P, kp, kh, rows, spp, nitems;  // the tuple's system
};

// One slice of A times the slices of B that still give a kept level: result
// columns sa P .. 8 P - 1, above N = 256 by two MMAs of about half of them.
// NKK K steps (the run-time nkk of them where NKK is 0).
template <class F, int P, int SA, int NKK>
__device__ __forceinline__ void mma_slice(uint32_t on, uint32_t d, uint64_t ad, uint64_t bd, int nkk,
                                          uint32_t acc) {
  constexpr int n = ((F::S - SA) * P + 15) & ~15;
  constexpr int n1 = n <= 256 ? n : ((n >> 1) + 15) & ~15, n2 = n - n1;
  constexpr int kMax = NKK ? NKK : kKChunk / 16;
#pragma unroll
  for (int kk = 0; kk < kMax; ++kk)
    if (NKK || kk < nkk)
      mma_if(on, d + SA * P, ad + 2 * kk, bd + 2 * kk, F::idesc(n1), kk == 0 && SA == 0 ? acc : 1u);
  if constexpr (n2 > 0) {
#pragma unroll
    for (int kk = 0; kk < kMax; ++kk)
      if (NKK || kk < nkk)
        mma_if(on, d + SA * P + n1, ad + 2 * kk, bd + n1 * 8 + 2 * kk, F::idesc(n2),
                 kk == 0 && SA == 0 ? acc : 1u);
  }
}

// A K chunk: the slices of A from the ring, spp to a slot.
template <class F, int P, int SA, int NKK>
__device__ __forceinline__ bool mma_chunk(MmaRole &m, uint32_t d, uint64_t &ad, uint64_t bd,
                                          int nkk, uint32_t acc, int *status) {
  if constexpr (SA < F::S) {
    if (F::SPLIT ? SA == 0 : (SA & (m.spp - 1)) == 0) {
      if (!mbar_wait_warp(&m.afull[m.st], m.ph, status, kErrFull)) return false;
      tc_fence_after();
      ad = sdesc_sw128(0) + ((m.ring_a + (uint32_t)(m.st * m.aslot)) >> 4);
    }
    mma_slice<F, P, SA, NKK>(m.leader, d, ad, bd, nkk, acc);
    ad += (uint32_t)(m.rows * 8);
    if (F::SPLIT ? SA == F::S - 1 : (SA & (m.spp - 1)) == m.spp - 1) {
      commit_if(m.leader, &m.aempty[m.st]);
      if (++m.st == m.nslots) {
        m.st = 0;
        m.ph ^= 1u;
      }
    }
    return mma_chunk<F, P, SA + 1, NKK>(m, d, ad, bd, nkk, acc, status);
  }
  return true;
}

// All items of a tuple.  The column count P is a template parameter so that
// every MMA's column offset and instruction descriptor are constants: a warp
// needs ~5 cycles for each instruction between two MMAs of 50 to 130.
template <class F, int P>
__device__ __forceinline__ bool mma_tuple(MmaRole &m, bool fresh, int *status) {
  constexpr int bufcols = F::S * P + (P & 8), nbuf = 2 * bufcols <= 512 ? 2 : 1;
  for (int it = 0; it < m.nitems; ++it, ++m.item) {
    // barrier `item & 1` serves every second item, whichever columns the
    // item has: its use u is item 2u + (item & 1)
    const int bb = m.item & 1, buf = nbuf == 2 ? bb : 0;
    const uint32_t u = m.item >> 1;
    if (u > 0 && !mbar_wait_warp(&m.acce[bb], (u - 1) & 1, status, kErrAccEmpty)) return false;
    if ((nbuf == 1 || (it == 0 && fresh)) && m.item > 0) {
      // one accumulator, or another layout than the item before had: that
      // item must be drained too
      const uint32_t p = m.item - 1;
      if (!mbar_wait_warp(&m.acce[p & 1], (p >> 1) & 1, status, kErrAccEmpty)) return false;
    }
    tc_fence_after();
    const uint32_t d = m.tm + buf * bufcols;
    uint32_t acc = 0;
    constexpr int parts = TcParts<F::CPLX>::kCount / F::PIECES;
    const int pt0 = F::PIECES == 2 && (it & 1) ? parts : 0;
    for (int pt = pt0; pt < pt0 + parts; ++pt) {
      const int K = TcParts<F::CPLX>::hole(pt) ? m.kh : m.kp;
      for (int k0 = 0; k0 < K; k0 += kKChunk) {
        const uint64_t bd = sdesc_sw128(0) + ((m.ring_b + (uint32_t)(m.bs * m.bslot)) >> 4);
        uint64_t ad = 0;
        const int nkk = (min(kKChunk, K - k0) + 15) / 16;
        const bool ok = nkk == 4 ? mma_chunk<F, P, 0, 4>(m, d, ad, bd, 4, acc, status)
                                 : mma_chunk<F, P, 0, 0>(m, d, ad, bd, nkk, acc, status);
        if (!ok) return false;
        acc = 1;
        if (++m.bs == m.nbslots) m.bs = 0;
      }
    }
    commit_if(m.leader, &m.accf[bb]);
  }
  return true;
}

template <class F>
__global__ void __launch_bounds__(kThreads, 1) triples_tc_kernel(const TcArgs g) {
  constexpr bool CPLX = F::CPLX;
  constexpr int S = F::S;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char *smem = reinterpret_cast<unsigned char *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char *ring = smem;
  unsigned char *bring = ring + g.nslots * g.aslot;
  unsigned char *tail = bring + g.nbslots * g.bslot;
  uint64_t *afull = reinterpret_cast<uint64_t *>(tail);
  uint64_t *aempty = afull + kMaxSlots;
  uint64_t *accf = aempty + kMaxSlots;
  uint64_t *acce = accf + 2;
  uint64_t *tfull = acce + 2;
  uint64_t *tempty = tfull + kTupleSlots;
  uint64_t *wfull = tempty + kTupleSlots;
  uint64_t *wfree = wfull + 2;
  uint64_t *drain = wfree + 2;
  uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(drain + 1);
  TcSlot *tslot = reinterpret_cast<TcSlot *>(tail + 448);
  double *ta = reinterpret_cast<double *>(tail + 576);
  double *tb = ta + kT1, *tc = tb + kT1, *red = tc + kT1;  // complex: (re, im) pairs
  static_assert((2 * kMaxSlots + 4 + 2 * kTupleSlots + 5) * 8 + 8 <= 448, "tail");
  static_assert(kTupleSlots * sizeof(TcSlot) <= 128, "tuple slots");

  int *status = g.flags;
  const int warp = uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < g.nslots; ++s) {
      mbar_init(&afull[s], 1);
      mbar_init(&aempty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&accf[b], 1);
      mbar_init(&acce[b], 128);
      mbar_init(&wfull[b], 1);
      mbar_init(&wfree[b], 1);
    }
    for (int s = 0; s < kTupleSlots; ++s) {
      mbar_init(&tfull[s], 1);
      mbar_init(&tempty[s], 3);
      tslot[s].t = -1;  // read, not used, where a wait for a tuple runs out
      tslot[s].s = 0;
    }
    mbar_init(drain, 1);
    fence_mbar_init();
  }
  // rows that no load writes (past a system's box, past the last stack row)
  // feed accumulator rows and columns nobody reads: any finite value will do
  for (int i = threadIdx.x; i < (g.nslots * g.aslot + g.nbslots * g.bslot) / 16; i += kThreads)
    reinterpret_cast<uint4 *>(ring)[i] = make_uint4(0, 0, 0, 0);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (warp == 1) {
    tmem_alloc(tmem_holder, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_holder;
  const size_t cells = (size_t)g.lay_cells;
  constexpr int kComp = CPLX ? 2 : 1;
  // a W cell: the level sums joined exactly -- (high, low) halves of levels
  // 0..3 and 4..7, or all levels of a split form in one integer
  using Cell = typename std::conditional<F::SPLIT, long long, longlong2>::type;
  Cell *planes =
      static_cast<Cell *>(g.planes) + (size_t)blockIdx.x * 2 * g.lay_pass * 3 * kComp * cells;

  if (warp == 0) {
    // ------------------------------------------------------ TMA producer
    const bool leader = elect_one();
    int st = 0, bs = 0;
    uint32_t use = 0;
    int cur = -1;
    int64_t cur_hi = 0;
    bool alive = true;
    const uint32_t ring_a = uniform(smem_u32(ring)), ring_b = uniform(smem_u32(bring));
    const TcDesc *d = g.sys;
    int kp = 0, kh = 0, rows = 0, ntiles = 0, npass = 0, spp = 0;
    uint32_t a_bytes = 0, b_bytes = 0;
    // queue positions are claimed g.claim at a time; a claim's tuples are
    // looked up together, one to a lane
    int64_t q0 = 0, pos = 0;
    int have = 0, next = 0;
    uint32_t packed = 0;
    // its status ends the other roles' first waits
    if (g.unpublished != 0) mbar_wait_warp(&tfull[0], 0, status, kErrFull, g.unpublished);
    for (uint32_t k = 0; g.unpublished == 0; ++k) {
      const int ts = k % kTupleSlots;
      const uint32_t tuse = k / kTupleSlots;
      if (tuse > 0 && !mbar_wait_warp(&tempty[ts], (tuse - 1) & 1, status, kErrEmpty))
        alive = false;
      if (next == have) {
        q0 = g.total;
        if (alive && leader && *reinterpret_cast<volatile int *>(status) == 0)
          q0 = (int64_t)atomicAdd(g.queue, (unsigned long long)g.claim);
        q0 = __shfl_sync(0xffffffffu, q0, __ffs(__ballot_sync(0xffffffffu, leader)) - 1);
        have = q0 >= g.total ? 0 : (int)min((int64_t)g.claim, g.total - q0);
        next = 0;
        if (lane < have) {
          const int64_t q = q0 + lane;
          int lo = max(cur, 0);  // queue positions only grow: walk on from the last system
          while (lo + 1 < g.nsys && g.prefix[lo + 1] <= q) ++lo;
          pos = g.sys[lo].t_begin + (g.order ? (int64_t)g.order[q] : q - g.prefix[lo]);
          packed = g.sys[lo].tuples[pos];
        }
        __syncwarp();
      }
      const bool stop = next == have || !alive;
      TcSlot s;
      s.a = s.b = s.c = s.s = 0;
      s.t = -1;
      if (!stop) {
        const int64_t q = q0 + next;
        if (q >= cur_hi) {
          int lo = max(cur, 0);
          while (lo + 1 < g.nsys && g.prefix[lo + 1] <= q) ++lo;
          cur = uniform(lo);
          cur_hi = g.prefix[cur + 1];
          d = g.sys + cur;
          const int nm = d->use_j ? kMaps : kMapsMain;
          for (int i = 0; i < nm; ++i) tensormap_acquire(&d->maps.Ta[0][0] + i);
          kp = uniform(d->Nv);
          kh = uniform(d->No);
          rows = uniform(d->rows);
          ntiles = (kh * kh + rows - 1) / rows;
          npass = uniform(d->use_j) ? 2 : 1;
          spp = uniform(d->spp);
          a_bytes = spp * rows * 128;
          b_bytes = S * uniform(d->P) * 128;
        }
        s.s = cur;
        s.t = __shfl_sync(0xffffffffu, pos, next);
        const int pk = __shfl_sync(0xffffffffu, (int)packed, next);
        ++next;
        s.a = pk & 0x3ff;
        s.b = (pk >> 10) & 0x3ff;
        s.c = (pk >> 20) & 0x3ff;
      }
      if (leader) {
        tslot[ts] = s;
        mbar_arrive(&tfull[ts]);
      }
      __syncwarp();
      if (stop) break;
      for (int gi = 0; gi < 3 * npass && alive; ++gi)
        for (int mt = 0; mt < ntiles && alive; ++mt)
          for (int pt = 0; pt < TcParts<CPLX>::kCount && alive; ++pt) {
            const TcPart p = part_of<CPLX>(d->maps, gi % 3, pt, s.a, s.b, s.c, gi / 3);
            const int K = TcParts<CPLX>::hole(pt) ? kh : kp;
            const int c2 = CPLX ? p.blk : p.bz, c3 = CPLX ? p.by * kp + p.bz : p.by;
            for (int k0 = 0; k0 < K && alive; k0 += kKChunk) {
#pragma unroll 1
              for (int sa = 0; sa < S; sa += spp) {
                if (use > 0 && !mbar_wait_warp(&aempty[st], (use - 1) & 1, status, kErrEmpty)) {
                  alive = false;
                  break;
                }
                if (leader) {
                  mbar_arrive_expect_tx(&afull[st], sa == 0 ? a_bytes + b_bytes : a_bytes);
                  // the chunk's B stack comes with its first A slot; its ring
                  // is one chunk deeper than A's, so that slot is free too
                  if (sa == 0)
                    tma_load_5d(ring_b + (uint32_t)(bs * g.bslot), p.bmap, &afull[st], k0, 0, c2, c3, 0);
                  tma_load_4d(ring_a + (uint32_t)(st * g.aslot), p.amap, &afull[st], k0, mt * rows,
                              p.ax, sa);
                }
                __syncwarp();
                if (++st == g.nslots) {
                  st = 0;
                  ++use;
                }
              }
              if (++bs == g.nbslots) bs = 0;
            }
          }
    }
    if (leader) {  // after a wait that gave up, here or elsewhere: copies in flight land first
      for (int i = 0; i < g.nslots; ++i) {
        const uint32_t n = use + (i < st ? 1 : 0);
        if (n > 0) mbar_drain(&afull[i], (n - 1) & 1);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // -------------------------------------------------------- MMA issuer
    const bool leader = elect_one();
    MmaRole m;
    m.st = m.bs = 0;
    m.ph = m.item = 0;
    m.nslots = g.nslots;
    m.nbslots = g.nbslots;
    m.aslot = g.aslot;
    m.bslot = g.bslot;
    m.ring_a = uniform(smem_u32(ring));
    m.ring_b = uniform(smem_u32(bring));
    m.tm = uniform(tmem);
    m.afull = afull;
    m.aempty = aempty;
    m.accf = accf;
    m.acce = acce;
    m.leader = leader;
    int prev = -1;
    bool alive = true;
    for (uint32_t k = 0; alive; ++k) {
      const int ts = k % kTupleSlots;
      if (!mbar_wait_warp(&tfull[ts], (k / kTupleSlots) & 1, status, kErrFull)) break;
      const bool stop = __any_sync(0xffffffffu, tslot[ts].t < 0);
      const int sys = uniform(tslot[ts].s);
      __syncwarp();
      if (leader) mbar_arrive(&tempty[ts]);
      if (stop) break;
      const TcDesc &d = g.sys[sys];
      const bool fresh = sys != prev;  // its accumulators may lie elsewhere
      prev = sys;
      if (fresh) {
        m.P = uniform(d.P);
        m.kp = uniform(d.Nv);
        m.kh = uniform(d.No);
        m.rows = uniform(d.rows);
        m.spp = uniform(d.spp);
        m.nitems =
            3 * (uniform(d.use_j) ? 2 : 1) * ((m.kh * m.kh + m.rows - 1) / m.rows) * F::PIECES;
      }
      if constexpr (CPLX) {  // P = 2 round_up(No, 8)
        switch (m.P) {
          case 16: alive = mma_tuple<F, 16>(m, fresh, status); break;
          case 32: alive = mma_tuple<F, 32>(m, fresh, status); break;
          case 48: alive = mma_tuple<F, 48>(m, fresh, status); break;
          default: alive = mma_tuple<F, 64>(m, fresh, status); break;
        }
      } else {
        switch (m.P) {
          case 8: alive = mma_tuple<F, 8>(m, fresh, status); break;
          case 16: alive = mma_tuple<F, 16>(m, fresh, status); break;
          case 24: alive = mma_tuple<F, 24>(m, fresh, status); break;
          case 32: alive = mma_tuple<F, 32>(m, fresh, status); break;
          case 40: alive = mma_tuple<F, 40>(m, fresh, status); break;
          case 48: alive = mma_tuple<F, 48>(m, fresh, status); break;
          case 56: alive = mma_tuple<F, 56>(m, fresh, status); break;
          default: alive = mma_tuple<F, 64>(m, fresh, status); break;
        }
      }
    }
    // no MMA outlives this role (after a failed wait some may be in flight)
    if (leader) {
      mma_commit(drain);
      mbar_drain(drain, 0);
    }
    __syncwarp();
  } else if (warp >= 4 && warp < 8) {
    // ------------------------------------------------ epilogue (4 warps)
    const int quarter = warp - 4;
    const int l = quarter * 32 + lane;
    uint32_t item = 0;
    bool alive = true;
    for (uint32_t k = 0; alive; ++k) {
      const int ts = k % kTupleSlots;
      bool ok = mbar_wait(&tfull[ts], (k / kTupleSlots) & 1, status, kErrFull);
      const int64_t t = tslot[ts].t;
      const int sys = tslot[ts].s;
      const TcDesc &d = g.sys[sys];
      uint32_t over = 0;
      ok = bar_and(1, 128, ok);
      if (threadIdx.x == 128) mbar_arrive(&tempty[ts]);
      if (!ok || t < 0) break;
      const int No = d.No, No2 = No * No, P = d.P, rows = d.rows;
      const int ntiles = (No2 + rows - 1) / rows, npass = d.use_j ? 2 : 1;
      const int bufcols = S * P + (P & 8), nbuf = 2 * bufcols <= 512 ? 2 : 1;
      const int wb = k & 1;
      const uint32_t wuse = k >> 1;
      ok = wuse == 0 || mbar_wait(&wfree[wb], (wuse - 1) & 1, status, kErrEmpty);
      for (int it = 0; it < 3 * npass * ntiles * F::PIECES; ++it, ++item) {
        const int tile = it / F::PIECES;
        const bool second = F::PIECES == 2 && (it & 1);  // added to what the first stored
        const int gi = tile / ntiles, mt = tile - gi * ntiles, grp = gi % 3, pass = gi / 3;
        Cell *plane0 = planes + (size_t)((wb * g.lay_pass + pass) * 3 + grp) * kComp * cells;
        const int bb = item & 1, buf = nbuf == 2 ? bb : 0;
        bool okw = ok && alive && mbar_wait(&accf[bb], (item >> 1) & 1, status, kErrAccFull);
        okw = bar_and(1, 128, okw);
        if (!okw) {
          alive = false;
          break;
        }
        tc_fence_after();
        const uint32_t tbase = tmem + ((uint32_t)(quarter * 32) << 16) + buf * bufcols;
        const int m = mt * rows + l;
        const bool valid = l < rows && m < No2;
        const int P1 = P / kComp;
        for (int cc = 0; cc < kComp * No;) {
          // column block (component) and its next 8 columns
          const int comp = kComp == 2 && cc >= No ? 1 : 0, c0 = cc - comp * No;
          cc += min(8, No - c0);
          Cell *plane = plane0 + comp * cells;
          float v[S][8];
          __syncwarp();
#pragma unroll
          for (int L = 0; L < S; ++L) tmem_ld8(tbase + L * P + comp * P1 + c0, v[L]);
          tmem_wait_ld();
          if (cc == kComp * No) {  // everything is read: the accumulator is free
            tc_fence_before();
            mbar_arrive(&acce[bb]);
          }
#pragma unroll
          for (int x = 0; x < 8; ++x) {
            const int r = c0 + x;
            if constexpr (F::SPLIT) {
              if (r < No && valid) {
                long long n = F::level(0, v[0][x]);
#pragma unroll
                for (int L = 1; L < S; ++L)
                  n = n * F::radix() + F::level(L, v[L][x]);
                plane[(size_t)r * No2 + m] = n;
              }
            } else if (r < No && valid) {
              // |level sum| < 2^22 for L >= 1 (flagged otherwise): adding
              // 1.5 2^23 leaves the integer n in the low mantissa bits b =
              // n + kBits.  Pairs of levels join in 32 bits (256 n + n' <
              // 2^31; the kBits cancel modulo 2^32), pairs of pairs in 64.
              constexpr uint32_t kBits = 0x4B400000u;
              uint32_t b[S];
#pragma unroll
              for (int L = 1; L < S; ++L) {
                b[L] = __float_as_uint(v[L][x] + 12582912.f);
                over |= b[L] ^ 0x4B000000u;  // exponent bits differ outside that range
              }
              const int n1 = (int)(b[1] - kBits);
              const int n23 = (int)(b[2] * 256u + b[3] - kBits * 257u);
              const int n45 = (int)(b[4] * 256u + b[5] - kBits * 257u);
              const int n67 = (int)(b[6] * 256u + b[7] - kBits * 257u);
              long long hi = (long long)__float2int_rn(v[0][x]) * (1 << 24) +
                             ((long long)n1 * 65536 + n23);
              long long lo = (long long)n45 * 65536 + n67;
              Cell &w = plane[(size_t)r * No2 + m];
              if (second) {  // stored by this thread
                hi += w.x;
                lo += w.y;
              }
              w = make_longlong2(hi, lo);
            }
          }
        }
      }
      if (!alive) break;
      __threadfence_block();
      bar_sync(1, 128);
      if (threadIdx.x == 128) mbar_arrive(&wfull[wb]);
      if (over & 0xFF800000u) atomicOr(&g.flags[1 + sys], 1);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------ energy (10 warps)
    const int er = ((warp < 4 ? warp - 2 : warp - 6) << 5) | lane;
    double *wd = g.wd + (size_t)blockIdx.x * g.lay_pass * kComp * cells;
    for (uint32_t k = 0;; ++k) {
      const int ts = k % kTupleSlots;
      bool ok = mbar_wait(&tfull[ts], (k / kTupleSlots) & 1, status, kErrFull);
      const TcSlot s = tslot[ts];
      ok = bar_and(2, kEnergyThreads, ok);
      if (er == 0) mbar_arrive(&tempty[ts]);
      if (!ok || s.t < 0) break;
      const TcDesc &d = g.sys[s.s];
      const int No = d.No, No2 = No * No;
      const int64_t Nv = d.Nv;
      const int a = s.a, b = s.b, c = s.c;
      // W, Z and the singles in units of a cell's high part (a power of two)
      const double inv = d.tai_sign / d.unit;
      if (er < No) {
#pragma unroll
        for (int h = 0; h < kComp; ++h) {
          ta[kComp * er + h] = d.tai[kComp * (a + er * Nv) + h] * inv;
          tb[kComp * er + h] = d.tai[kComp * (b + er * Nv) + h] * inv;
          tc[kComp * er + h] = d.tai[kComp * (c + er * Nv) + h] * inv;
        }
      }
      const int wb = k & 1;
      ok = mbar_wait(&wfull[wb], (k >> 1) & 1, status, kErrAccFull);
      const int npass = d.use_j ? 2 : 1;
      // x / n = umulhi(x, by_n) for x < 2^18 and 2 <= n <= 64
      const uint32_t by_no = 0xffffffffu / (uint32_t)No + 1u;
      const uint32_t by_ti = 0xffffffffu / (uint32_t)((No + 7) >> 3) + 1u;
      const uint32_t by_tj = 0xffffffffu / (uint32_t)((No + 3) >> 2) + 1u;
      for (int pc = 0; pc < npass * kComp; ++pc) {
        const int pass = pc / kComp, comp = pc % kComp;
        const Cell *p0 =
            planes + (size_t)((wb * g.lay_pass + pass) * 3 * kComp + comp) * cells;
        const Cell *p1 = p0 + kComp * cells, *p2 = p1 + kComp * cells;
        double *W = wd + pc * cells;
        // a warp takes 8 x 4 elements (i,j) of one k: every plane's cells then
        // come in whole 32-byte sectors (group 2's run along j); No=37/Nv=151
        // with (cT) 8.4 -> 8.0 ms, No=24/Nv=240 in 3 BF16 slices 9.0 -> 8.4 ms.
        // Few orbitals, whose cells stay in L2 and fill such tiles badly, are
        // taken in order (No=4..20: tiles 2 % slower; together with the order of
        // the triples, No=21..24 and Nv=60..200: No=24 in order 6 to 18 % slower,
        // No=22 FP64 5 to 7 % slower and 3 slices 1 to 2 % faster, No=21, 23 FP64
        // 1 to 2 % faster and 3 slices 3 to 8 % slower)
        constexpr int kU = 4;
        const bool tiled = No > 20;
        const int ti = tiled ? (No + 7) >> 3 : 1, tj = (No + 3) >> 2;
        const int tiles = tiled ? ti * tj * No : (No * No2 + 31) >> 5;
        for (int t0 = er >> 5; t0 < tiles; t0 += kU * kEnergyWarps) {
          Cell v[kU][3];
          int at[kU];
#pragma unroll
          for (int u = 0; u < kU; ++u) {
            const int t = t0 + u * kEnergyWarps;
            int i, j, kx;
            if (tiled) {
              const int r = (int)__umulhi((uint32_t)t, by_ti);
              kx = (int)__umulhi((uint32_t)r, by_tj);
              i = (t - r * ti) * 8 + (lane & 7);
              j = (r - kx * tj) * 4 + (lane >> 3);
            } else {
              const int idx = t * 32 + lane, jk = (int)__umulhi((uint32_t)idx, by_no);
              i = idx - jk * No;
              kx = (int)__umulhi((uint32_t)jk, by_no);
              j = jk - kx * No;
            }
            at[u] = t < tiles && i < No && j < No && kx < No ? i + No * j + No2 * kx : -1;
            if (at[u] >= 0) {
              v[u][0] = p0[at[u]];
              v[u][1] = p1[j * No2 + i + No * kx];
              v[u][2] = p2[i * No2 + j + No * kx];
            }
          }
#pragma unroll
          for (int u = 0; u < kU; ++u) {
            const int idx = at[u];
            if (idx >= 0) {
              if constexpr (F::SPLIT) {  // below 2^50: exact
                W[idx] = i64_to_f64(v[u][0] + v[u][1] + v[u][2]);
              } else {
                // both sums are exact; one rounding where they are joined
                const long long hi = v[u][0].x + v[u][1].x + v[u][2].x;
                const long long lo = v[u][0].y + v[u][1].y + v[u][2].y;
                W[idx] = fma(i64_to_f64(lo), 0x1p-32, i64_to_f64(hi));
              }
            }
          }
        }
      }
      __threadfence_block();
      bar_sync(2, kEnergyThreads);
      if (er == 0) mbar_arrive(&wfree[wb]);
      int cls = 0;  // src/atrip/Atrip.cxx:640-642
      if (a == b) cls++;
      if (b == c) cls--;
      const double epsabc = d.epsa[kComp * a] + d.epsa[kComp * b] + d.epsa[kComp * c];
      const double *Vbc = d.Vhh + ((int64_t)b * Nv + c) * No2 * kComp;
      const double *Vac = d.Vhh + ((int64_t)a * Nv + c) * No2 * kComp;
      const double *Vab = d.Vhh + ((int64_t)a * Nv + b) * No2 * kComp;
      double en[2];
      for (int pass = 0; pass < npass; ++pass) {
        double sum = 0.0;
        if constexpr (CPLX) {
          const TcSinglesZ sc = {
              reinterpret_cast<const double2 *>(Vbc), reinterpret_cast<const double2 *>(Vac),
              reinterpret_cast<const double2 *>(Vab), reinterpret_cast<const double2 *>(ta),
              reinterpret_cast<const double2 *>(tb), reinterpret_cast<const double2 *>(tc)};
          if (ok)
            sum = energy_partial_z(d, wd + pass * 2 * cells, wd, cells, sc, cls == 0, epsabc, er);
        } else {
          const TcSinglesCtx sc = {Vbc, Vac, Vab, ta, tb, tc};
          if (ok) sum = energy_partial<F::SPLIT>(d, wd + pass * cells, wd, sc, cls == 0, epsabc, er);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) red[er >> 5] = sum;
        bar_sync(2, kEnergyThreads);
        double e = 0.0;
        for (int w = 0; w < kEnergyWarps; ++w) e += red[w];
        bar_sync(2, kEnergyThreads);  // red, ta.. and wd are reused
        en[pass] = e * d.unit * (pass ? d.unit_j : d.unit);
      }
      if (er == 0) {
        d.e[s.t] = en[0];
        d.ect[s.t] = npass == 2 ? en[1] : en[0];
      }
    }
    __syncwarp();
  }
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

// ------------------------------------------------------------------ prep

// The largest magnitude of x[0 .. n), as an FP64 bit pattern (ordered like the
// magnitudes; infinities and NaN sort above every finite value).
__global__ void __launch_bounds__(256) max_kernel(const double *__restrict__ x, int64_t n,
                                                  unsigned long long *__restrict__ out) {
  unsigned long long m = 0;
  for (int64_t i = blockIdx.x * 256ll + threadIdx.x; i < n; i += gridDim.x * 256ll) {
    const unsigned long long b = magnitude(x[i]);
    m = b > m ? b : m;
  }
  warp_max(m, out);
}

// The profile of T: t[E][x] = log of max |Ta[x][q][p][E]|, and the largest.
template <int NC>
__global__ void __launch_bounds__(256) t_profile_kernel(const double *__restrict__ Ta, int No2,
                                                        int Nv, int *__restrict__ t,
                                                        unsigned long long *__restrict__ out) {
  __shared__ unsigned long long sh[8][32];
  const int x = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int E = blockIdx.y * 32 + lane;
  unsigned long long m = 0;
  if (E < Nv) {
    const double *p = Ta + ((int64_t)x * No2 * Nv + E) * NC;
#pragma unroll 4
    for (int r = warp; r < No2; r += 8)
#pragma unroll
      for (int h = 0; h < NC; ++h) {
        const unsigned long long b = magnitude(p[(int64_t)r * Nv * NC + h]);
        m = b > m ? b : m;
      }
  }
  sh[warp][lane] = m;
  __syncthreads();
  if (warp != 0) return;
  for (int w = 1; w < 8; ++w) m = sh[w][lane] > m ? sh[w][lane] : m;
  if (E < Nv) t[(size_t)E * profile_pitch(Nv) + x] = log_of(m);
  warp_max(m, out);
}

// The least product of T's profile with those of 32 slabs Vpt[y][z][r][E] a
// block (FULL: exact, else a lower bound), and the largest element.  Reads V
// once; the slab maxima it replaces read as much (No=24/Nv=240, first run of 8000
// tuples with examination and cut: 15.2 ms with either, 15.6 with the exact
// products).
template <int NC, bool FULL>
__global__ void __launch_bounds__(256) v_profile_kernel(const double *__restrict__ Vpt,
                                                        const int *__restrict__ t, int No, int Nv,
                                                        unsigned long long *__restrict__ vmax,
                                                        unsigned int *__restrict__ least) {
  extern __shared__ int v[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t p0 = (int64_t)blockIdx.x * kProfilePairs, np = (int64_t)Nv * Nv;
  unsigned long long best = 0;
  for (int k = warp; k < kProfilePairs; k += 8)
    for (int E = lane; E < Nv; E += 32) {
      unsigned long long m = 0;
      if (p0 + k < np) {
        const double *p = Vpt + ((p0 + k) * No * Nv + E) * NC;
#pragma unroll 8
        for (int r = 0; r < No; ++r)
#pragma unroll
          for (int h = 0; h < NC; ++h) {
            const unsigned long long b = magnitude(p[(int64_t)r * Nv * NC + h]);
            m = b > m ? b : m;
          }
      }
      v[E * (kProfilePairs + 1) + k] = log_of(m);
      best = m > best ? m : best;
    }
  warp_max(best, vmax);
  __syncthreads();
  least_product<FULL>(t, v, Nv, p0, least);
}

// dst[s][R][k] (pitch Kp) = digit_s(sign src(R, k)), row R = (o n1 + r1) n2
// + r2.  norms[s], s < kNormSlices: the largest row sum of q_s^2.
struct CutJob {
  const double *src;
  __nv_bfloat16 *dst;
  int64_t nrows, n1, n2, so, s1, s2, sk;
  int K, Kp, e, neg;
  unsigned int *norms;
  int nblk = 1, blk = 0;  // dst holds nblk blocks of n2 rows for each of src's: this is block blk
};

__global__ void __launch_bounds__(256) cut_kernel(CutJob j) {
  const int64_t plane = j.nrows * j.nblk * j.Kp;
  const int lane = threadIdx.x & 31;
  const int64_t nw = (int64_t)gridDim.x * 8;
  unsigned int best[kNormSlices] = {};
  for (int64_t R = blockIdx.x * 8 + (threadIdx.x >> 5); R < j.nrows; R += nw) {
    const int64_t r2 = R % j.n2, t = R / j.n2, r1 = t % j.n1, o = t / j.n1;
    const double *src = j.src + o * j.so + r1 * j.s1 + r2 * j.s2;
    __nv_bfloat16 *dst = j.dst + ((t * j.nblk + j.blk) * j.n2 + r2) * j.Kp;
    float nrm[kNormSlices] = {};  // whole numbers below 2^24
    for (int k = 2 * lane; k < j.Kp; k += 64) {
      unsigned long long y[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        long long X = k + h < j.K ? fixed63(src[(k + h) * j.sk], j.e) : 0;
        if (j.neg) X = -X;
        y[h] = biased(X);
      }
#pragma unroll
      for (int s = 0; s < kS; ++s) {
        float q[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          q[h] = digit(y[h], s);
          if (s < kNormSlices) nrm[s] = fmaf(q[h], q[h], nrm[s]);
        }
        *reinterpret_cast<__nv_bfloat162 *>(dst + s * plane + k) =
            __floats2bfloat162_rn(q[0], q[1]);
      }
    }
#pragma unroll
    for (int s = 0; s < kNormSlices; ++s) {
      const unsigned int v = __reduce_add_sync(0xffffffffu, (unsigned int)nrm[s]);
      best[s] = v > best[s] ? v : best[s];
    }
  }
  unsigned int v = 0;  // lane s takes digit s
#pragma unroll
  for (int s = 0; s < kNormSlices; ++s)
    if (lane == s) v = best[s];
  if (lane < kNormSlices && v > *(volatile unsigned int *)&j.norms[lane])
    atomicMax(&j.norms[lane], v);
}

// ------------------------------------------------------------------ host

struct TcImpl {
  int S = kS;
  bool split = false, f16 = false;
  int nc = 1;  // doubles per element: 2 for a complex system
  int No = 0, Nv = 0, P = 0, rows = 0, spp = 0, Kp = 0, Kh = 0;
  int eT = 0, eV = 0, eJ = 0;
  DigitNorms nT, nU;            // of the T rows (over E; over L)
  int pieces = 1, pieces_j = 1;
  double unit = 1.0, unit_j = 1.0;
  char *arena = nullptr, *arena_j = nullptr;
  TcMaps maps;
};

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }();
  return fn;
}

// BF16 tensor map of `rank` dimensions, K fastest, 128-byte swizzle.  The K
// extent is the padded one, whole chunks: a box that leaves the tensor in its
// innermost dimension takes ~7 cycles a row (18 B per cycle), one inside it
// 1.1 (119 B per cycle); rows past the other extents cost nothing extra.
int make_map(CUtensorMap *m, void *base, int rank, const uint64_t *dims, const uint32_t *box) {
  auto fn = encode_fn();
  if (!fn) {
    set_error("cuTensorMapEncodeTiled not available from the driver");
    return ATRIP_ERR_CUDA;
  }
  uint64_t strides[4], s = dims[0] * 2;
  for (int i = 1; i < rank; ++i) {
    strides[i - 1] = s;
    s *= dims[i];
  }
  const uint32_t one[5] = {1, 1, 1, 1, 1};
  const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, base, dims, strides, box, one,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed with CUresult " + std::to_string((int)r));
    return ATRIP_ERR_CUDA;
  }
  return ATRIP_OK;
}

int map_a(CUtensorMap *m, void *base, const TcImpl &p, int K) {
  const uint64_t d[4] = {(uint64_t)K, (uint64_t)p.No * p.No, (uint64_t)p.Nv,
                         (uint64_t)p.S};
  const uint32_t box[4] = {kKChunk, (uint32_t)p.rows, 1, (uint32_t)p.spp};
  return make_map(m, base, 4, d, box);
}
int map_b(CUtensorMap *m, void *base, const TcImpl &p, int K) {
  if (p.nc == 2) {  // (K, r, block, (y,z), slice): two neighbouring column blocks of three
    const uint64_t d[5] = {(uint64_t)K, (uint64_t)p.No, kBlocksZ, (uint64_t)p.Nv * p.Nv, kS};
    const uint32_t box[5] = {kKChunk, (uint32_t)p.P / 2, 2, 1, kS};
    return make_map(m, base, 5, d, box);
  }
  const uint64_t d[5] = {(uint64_t)K, (uint64_t)p.No, (uint64_t)p.Nv, (uint64_t)p.Nv,
                         (uint64_t)p.S};
  const uint32_t box[5] = {kKChunk, (uint32_t)p.P, 1, 1, (uint32_t)p.S};
  return make_map(m, base, 5, d, box);
}

// Smallest e with x <= 127/128 2^e (the top digit then stays below 128).
int exponent_of(double x) {
  int e = std::ilogb(x) + 1;
  if (x > std::ldexp(127.0 / 128.0, e)) ++e;
  return e;
}

double as_double(unsigned long long b) {
  double d;
  std::memcpy(&d, &b, sizeof(d));
  return d;
}

struct DeviceStats {
  unsigned long long t_max, vp_max, vh_max;  // largest magnitudes
  unsigned int least[2];                     // least product (log_of sums): lower bound, exact
  unsigned int n[8][8];                      // digit norms of up to eight cut jobs
};

// Queue the examination of T against a pair V_hhhp, V_pphp (or J): maxima and
// the least product, or (FULL) only that, exact.  scratch: profile_bytes() of
// device memory.
template <int NC, bool FULL>
int examine(const double *Ta, const double *vht, const double *vpt, int No, int Nv, void *scratch,
            DeviceStats *ds, cudaStream_t st, int64_t *launches) {
  int *t = static_cast<int *>(scratch);
  if (!FULL) {
    t_profile_kernel<NC><<<dim3(Nv, (Nv + 31) / 32), 256, 0, st>>>(Ta, No * No, Nv, t, &ds->t_max);
    ATRIP_CUDA_TRY(cudaGetLastError());
  }
  auto kern = v_profile_kernel<NC, FULL>;
  ATRIP_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      kProfileSmem));
  kern<<<(unsigned)(((int64_t)Nv * Nv + kProfilePairs - 1) / kProfilePairs), 256, profile_smem(Nv),
         st>>>(vpt, t, No, Nv, &ds->vp_max, &ds->least[FULL]);
  ATRIP_CUDA_TRY(cudaGetLastError());
  *launches += 1;
  if (FULL) return ATRIP_OK;
  max_kernel<<<152 * 4, 256, 0, st>>>(vht, (int64_t)NC * Nv * No * No * No, &ds->vh_max);
  ATRIP_CUDA_TRY(cudaGetLastError());
  *launches += 2;
  return ATRIP_OK;
}

// Clear *ds, examine and read the result back (synchronises st).
bool grids_of(const DeviceStats &h, int *e_t, int *e_v, bool *loose);
int examine(int nc, const double *Ta, const double *vht, const double *vpt, int No, int Nv,
            void *scratch, DeviceStats *ds, DeviceStats *h, cudaStream_t st, int64_t *launches) {
  std::memset(h, 0, sizeof(*h));
  h->least[0] = h->least[1] = ~0u;
  ATRIP_CUDA_TRY(cudaMemcpyAsync(ds, h, sizeof(*h), cudaMemcpyHostToDevice, st));
  for (int full = 0; full < 2; ++full) {
    const auto run = nc == 2 ? (full ? examine<2, true> : examine<2, false>)
                             : (full ? examine<1, true> : examine<1, false>);
    const int rc = run(Ta, vht, vpt, No, Nv, scratch, ds, st, launches);
    if (rc != ATRIP_OK) return rc;
    ATRIP_CUDA_TRY(cudaMemcpyAsync(h, ds, sizeof(*h), cudaMemcpyDeviceToHost, st));
    ATRIP_CUDA_TRY(cudaStreamSynchronize(st));
    if (!full) h->least[1] = h->least[0];
    int e_t, e_v;
    bool loose = false;
    if (grids_of(*h, &e_t, &e_v, &loose) && loose) break;  // as good as it gets
  }
  return ATRIP_OK;
}

cudaError_t cut(CutJob j, cudaStream_t st) {
  const int grid = (int)std::min<int64_t>((j.nrows + 7) / 8, 152 * 8);
  cut_kernel<<<grid, 256, 0, st>>>(j);
  return cudaGetLastError();
}

size_t up(size_t x) { return (x + 1023) / 1024 * 1024; }

// The slices may take at most half of the memory that is free: the rest is
// the host program's.  false (no error) when they do not fit.  They are given
// back where the engine finds no memory for anything else (device_alloc), by
// atrip_gpu_trim and when an operand is uploaded anew.
bool alloc_arena(char **p, size_t bytes) {
  size_t fr = 0, tot = 0;
  if (cudaMemGetInfo(&fr, &tot) != cudaSuccess || bytes > fr / 2 ||
      cudaMalloc(p, bytes) != cudaSuccess) {
    cudaGetLastError();
    *p = nullptr;
    return false;
  }
  return true;
}

bool exponent_ok(int e) { return e >= -200 && e <= 200; }

// The grids' exponents, if an examination's result allows the form; *loose:
// loose level sums too.
bool grids_of(const DeviceStats &h, int *e_t, int *e_v, bool *loose) {
  const unsigned long long mT = h.t_max, mV = std::max(h.vp_max, h.vh_max);
  constexpr unsigned long long kInf = 0x7ff0000000000000ull;
  if (mT == 0 || mV == 0 || mT >= kInf || mV >= kInf) return false;
  *e_t = exponent_of(as_double(mT));
  *e_v = exponent_of(as_double(mV));
  if (!exponent_ok(*e_t) || !exponent_ok(*e_v)) return false;
  const double least = std::ldexp((double)h.least[1], -kLogOne) - 2 * kLogBias - (*e_t + *e_v);
  *loose = least >= -kLooseBits;
  return least >= -kRangeBits;
}

DigitNorms norms_of(const unsigned int *x) {
  DigitNorms n;
  for (int s = 0; s < kNormSlices; ++s) n.q2[s] = (double)x[s];
  return n;
}

// Accumulators a row tile's sums need to be exact: one for its natural and
// transposed half, or one each; 0: not exact either.  A complex system's rows
// meet real and imaginary columns.
int sum_pieces(int nc, const DigitNorms &nT, const DigitNorms &nV, const DigitNorms &nH,
               const DigitNorms &nU, bool loose) {
  return level_sums_exact(2 * nc, nT, nV, nH, nU, loose) ? 1
         : level_sums_exact(nc, nT, nV, nH, nU, loose)   ? 2
                                                         : 0;
}

// A column operand: its one block, or the three of a complex system, of
// components comp[] and signs.
int cut_blocks(const TcImpl &p, CutJob j, const int *comp, const int *neg, cudaStream_t st,
               int64_t *launches) {
  const double *src = j.src;
  j.nblk = p.nc == 2 ? kBlocksZ : 1;
  for (int b = 0; b < j.nblk; ++b) {
    j.blk = b;
    j.src = src + comp[b];
    j.neg = neg[b];
    ATRIP_CUDA_TRY(cut(j, st));
    *launches += 1;
  }
  return ATRIP_OK;
}

// A row operand, natural and transposed rows (r1 and r2 exchanged), one
// component after the other at dst[].
int cut_rows(const TcImpl &p, CutJob j, __nv_bfloat16 *const *dst, cudaStream_t st,
             int64_t *launches) {
  const double *src = j.src;
  for (int c = 0; c < p.nc; ++c)
    for (int tr = 0; tr < 2; ++tr) {
      j.src = src + c;
      j.dst = dst[2 * c + tr];
      ATRIP_CUDA_TRY(cut(j, st));
      std::swap(j.s1, j.s2);
      *launches += 1;
    }
  return ATRIP_OK;
}

constexpr int kCompV[kBlocksZ] = {1, 0, 1}, kNegV[kBlocksZ] = {1, 0, 0};
constexpr int kCompT[kBlocksZ] = {0, 1, 0}, kNegT[kBlocksZ] = {1, 1, 0};
constexpr int kReal[1] = {0}, kPos[1] = {0}, kNeg[1] = {1};

// Cut V_pphp / V_hhhp (or the J pair), scale 2^e shared by both.
int cut_pair(const TcImpl &p, const double *vht, const double *vpt, int e,
             __nv_bfloat16 *const *vh, __nv_bfloat16 *vp, DeviceStats *ds, cudaStream_t st,
             int64_t *launches) {
  const int64_t No = p.No, Nv = p.Nv, No2 = No * No, nc = p.nc;
  CutJob j;
  j.e = e;
  j.neg = 0;
  j.src = vht; j.nrows = Nv * No2; j.n1 = No; j.n2 = No;
  j.so = No2 * No * nc; j.s1 = No2 * nc; j.s2 = No * nc; j.sk = nc; j.K = p.No; j.Kp = p.Kh;
  j.norms = ds->n[4];
  const int rc = cut_rows(p, j, vh, st, launches);
  if (rc != ATRIP_OK) return rc;
  j.src = vpt; j.dst = vp; j.nrows = Nv * Nv * No; j.n1 = Nv; j.n2 = No;
  j.so = Nv * No * Nv * nc; j.s1 = No * Nv * nc; j.s2 = Nv * nc; j.sk = nc;
  j.K = p.Nv; j.Kp = p.Kp;
  j.norms = ds->n[5];
  return nc == 2 ? cut_blocks(p, j, kCompV, kNegV, st, launches)
                 : cut_blocks(p, j, kReal, kPos, st, launches);
}

void free_impl(TcImpl *p) {
  if (!p) return;
  cudaFree(p->arena);
  cudaFree(p->arena_j);
  delete p;
}

struct ScopedDevice {  // device allocation freed on scope exit
  void *p = nullptr;
  ~ScopedDevice() { cudaFree(p); }
};

// Rows of an item: the No^2 rows in equal shares of at most 128.
int item_rows(int No) {
  const int nt = (No * No + 127) / 128;
  return ((No * No + nt - 1) / nt + 7) / 8 * 8;
}

int prepare_main(TcState &s, const DeviceTensors &dt, int No_, int Nv_, bool cplx,
                 cudaStream_t st, int64_t *launches) {
  auto *p = new TcImpl();
  s.impl = p;
  p->nc = cplx ? 2 : 1;
  p->No = No_;
  p->Nv = Nv_;
  p->P = p->nc * ((No_ + 7) / 8 * 8);
  p->rows = item_rows(No_);
  // slices per copy (a ring slot): up to 32 KB.  A role's warp needs ~200
  // cycles for a wait and a signal whatever the size, so a slot should hold
  // several MMAs' work
  p->spp = p->rows > 104 ? 2 : 4;
  p->Kp = (Nv_ + kKChunk - 1) / kKChunk * kKChunk;
  p->Kh = kKChunk;
  const int64_t No = No_, Nv = Nv_, No2 = No * No, nc = p->nc, nblk = cplx ? kBlocksZ : 1;
  const size_t nTa = up((size_t)2 * kS * Nv * No2 * p->Kp), nVh = up((size_t)2 * kS * Nv * No2 * p->Kh),
               nVp = up((size_t)2 * kS * Nv * Nv * No * nblk * p->Kp),
               nTp = up((size_t)2 * kS * Nv * Nv * No * nblk * p->Kh);
  if (!alloc_arena(&p->arena, 2 * nc * (nTa + nVh) + nVp + 2 * nTp)) return ATRIP_OK;
  ScopedDevice tmp;
  ATRIP_CUDA_TRY(device_alloc(&tmp.p, sizeof(DeviceStats)));
  auto *ds = static_cast<DeviceStats *>(tmp.p);
  DeviceStats h;
  int rc = examine(p->nc, dt.Ta, dt.Vht, dt.Vpt, No_, Nv_, p->arena, ds, &h, st, launches);
  bool loose = false;
  if (rc != ATRIP_OK || !grids_of(h, &p->eT, &p->eV, &loose)) return rc;
  p->unit = std::ldexp(1.0, p->eT + p->eV - 14 - 24);

  char *q = p->arena;
  auto take = [&](size_t n) {
    char *r = q;
    q += n;
    return reinterpret_cast<__nv_bfloat16 *>(r);
  };
  __nv_bfloat16 *Ta[4], *Vh[4];
  for (int i = 0; i < 2 * nc; ++i) Ta[i] = take(nTa);
  for (int i = 0; i < 2 * nc; ++i) Vh[i] = take(nVh);
  __nv_bfloat16 *Vp = take(nVp), *TpN = take(nTp), *TpT = take(nTp);
  CutJob j;
  j.e = p->eT;
  j.neg = 0;
  // rows (p,q) of T_x over E, p fastest and q fastest
  j.src = dt.Ta; j.nrows = Nv * No2; j.n1 = No; j.n2 = No;
  j.so = No2 * Nv * nc; j.s1 = No * Nv * nc; j.s2 = Nv * nc; j.sk = nc; j.K = Nv_; j.Kp = p->Kp;
  j.norms = ds->n[0];
  rc = cut_rows(*p, j, Ta, st, launches);
  if (rc != ATRIP_OK) return rc;
  // columns r of -T[u,v,L,r] and -T[u,v,r,L] over L
  const int *comp = cplx ? kCompT : kReal, *neg = cplx ? kNegT : kNeg;
  j.src = dt.Tp; j.dst = TpN; j.nrows = Nv * Nv * No; j.n1 = Nv; j.n2 = No;
  j.so = Nv * No2 * nc; j.s1 = No2 * nc; j.s2 = No * nc; j.sk = nc; j.K = No_; j.Kp = p->Kh;
  j.norms = ds->n[1];
  if ((rc = cut_blocks(*p, j, comp, neg, st, launches)) != ATRIP_OK) return rc;
  j.dst = TpT; j.s2 = nc; j.sk = No * nc;
  j.norms = ds->n[2];
  if ((rc = cut_blocks(*p, j, comp, neg, st, launches)) != ATRIP_OK) return rc;
  rc = cut_pair(*p, dt.Vht, dt.Vpt, p->eV, Vh, Vp, ds, st, launches);
  if (rc != ATRIP_OK) return rc;
  ATRIP_CUDA_TRY(cudaMemcpyAsync(&h, ds, sizeof(h), cudaMemcpyDeviceToHost, st));
  ATRIP_CUDA_TRY(cudaStreamSynchronize(st));
  p->nT = norms_of(h.n[0]);
  p->nU = norms_of(h.n[1]);
  const DigitNorms nU2 = norms_of(h.n[2]);
  for (int s = 0; s < kNormSlices; ++s) p->nU.q2[s] = std::max(p->nU.q2[s], nU2.q2[s]);
  p->pieces = sum_pieces(p->nc, p->nT, norms_of(h.n[5]), norms_of(h.n[4]), p->nU, loose);
  if (p->pieces == 0) return ATRIP_OK;

  for (int i = 0; i < 4; ++i) {  // [component][row order]; a real system's twice
    const int k = i % (2 * nc);
    if ((rc = map_a(&p->maps.Ta[i / 2][i % 2], Ta[k], *p, p->Kp)) ||
        (rc = map_a(&p->maps.Vh[i / 2][i % 2], Vh[k], *p, p->Kh)))
      return rc;
  }
  if ((rc = map_b(&p->maps.Vp, Vp, *p, p->Kp)) || (rc = map_b(&p->maps.TpN, TpN, *p, p->Kh)) ||
      (rc = map_b(&p->maps.TpT, TpT, *p, p->Kh)))
    return rc;
  std::memcpy(p->maps.Jh, p->maps.Vh, sizeof(p->maps.Jh));
  p->maps.Jp = p->maps.Vp;
  s.usable = true;
  return ATRIP_OK;
}

int prepare_j(TcState &s, const DeviceTensors &dt, cudaStream_t st, int64_t *launches) {
  auto *p = static_cast<TcImpl *>(s.impl);
  const int64_t No = p->No, Nv = p->Nv, No2 = No * No, nc = p->nc;
  const int64_t nblk = nc == 2 ? kBlocksZ : 1;
  const size_t nVh = up((size_t)2 * kS * Nv * No2 * p->Kh),
               nVp = up((size_t)2 * kS * Nv * Nv * No * nblk * p->Kp);
  if (!alloc_arena(&p->arena_j, 2 * nc * nVh + nVp)) return ATRIP_OK;
  ScopedDevice tmp;
  ATRIP_CUDA_TRY(device_alloc(&tmp.p, sizeof(DeviceStats)));
  auto *ds = static_cast<DeviceStats *>(tmp.p);
  DeviceStats h;
  int e_t;
  int rc = examine((int)nc, dt.Ta, dt.Jht, dt.Jpt, p->No, p->Nv, p->arena_j, ds, &h, st, launches);
  bool loose = false;
  if (rc != ATRIP_OK || !grids_of(h, &e_t, &p->eJ, &loose)) return rc;
  p->unit_j = std::ldexp(1.0, p->eT + p->eJ - 14 - 24);
  __nv_bfloat16 *vh[4];
  for (int i = 0; i < 2 * nc; ++i) vh[i] = reinterpret_cast<__nv_bfloat16 *>(p->arena_j + i * nVh);
  auto *vp = reinterpret_cast<__nv_bfloat16 *>(p->arena_j + 2 * nc * nVh);
  rc = cut_pair(*p, dt.Jht, dt.Jpt, p->eJ, vh, vp, ds, st, launches);
  if (rc != ATRIP_OK) return rc;
  ATRIP_CUDA_TRY(cudaMemcpyAsync(&h, ds, sizeof(h), cudaMemcpyDeviceToHost, st));
  ATRIP_CUDA_TRY(cudaStreamSynchronize(st));
  const int pieces = sum_pieces(p->nc, p->nT, norms_of(h.n[5]), norms_of(h.n[4]), p->nU, loose);
  if (pieces == 0) return ATRIP_OK;
  p->pieces_j = std::max(p->pieces, pieces);
  for (int i = 0; i < 4; ++i)
    if ((rc = map_a(&p->maps.Jh[i / 2][i % 2], vh[i % (2 * nc)], *p, p->Kh))) return rc;
  if ((rc = map_b(&p->maps.Jp, vp, *p, p->Kp))) return rc;
  s.usable_j = true;
  return ATRIP_OK;
}

// Free what an unusable preparation left behind (the verdict stays).
void drop_impl(TcState &s) {
  free_impl(static_cast<TcImpl *>(s.impl));
  s.impl = nullptr;
  s.usable = s.usable_j = false;
}

}  // namespace

void tc_free(TcState &s) {
  if (s.impl) {
    drop_impl(s);
    s.generation++;
  }
  s.tried = s.tried_j = s.usable = s.usable_j = false;
}

// The line: the work of the system's whole list, so that every range of one
// system takes the same kernel.  Cutting the slices costs ~2 ms in
// allocations, launches and tensor maps the first time, about what the DFMA
// kernel needs for 1e9 FLOPs at these sizes (No=4/Nv=12, 4.5e6: 0.1 ms).
int tc_split_attach(TcState &s, int S, bool f16, int No, int Nv, int Kp, double unit,
                    void *const *ops) {
  tc_free(s);
  auto *p = new TcImpl();
  s.impl = p;
  p->S = S;
  p->split = true;
  p->f16 = f16;
  p->No = No;
  p->Nv = Nv;
  p->P = (No + 7) / 8 * 8;
  p->rows = item_rows(No);
  p->spp = S;
  p->Kp = Kp;
  p->Kh = kKChunk;
  // level 0 of a cell carries S - 1 radices more
  p->unit = std::ldexp(unit, -(f16 ? 11 : 8) * (S - 1));
  int rc;
  for (int i = 0; i < 4; ++i)
    if ((rc = map_a(&p->maps.Ta[i / 2][i % 2], ops[i % 2], *p, p->Kp)) ||
        (rc = map_a(&p->maps.Vh[i / 2][i % 2], ops[2 + i % 2], *p, p->Kh)))
      return rc;
  if ((rc = map_b(&p->maps.Vp, ops[4], *p, p->Kp)) || (rc = map_b(&p->maps.TpN, ops[5], *p, p->Kh)) ||
      (rc = map_b(&p->maps.TpT, ops[6], *p, p->Kh)))
    return rc;
  std::memcpy(p->maps.Jh, p->maps.Vh, sizeof(p->maps.Jh));
  p->maps.Jp = p->maps.Vp;
  s.tried = s.usable = true;
  return ATRIP_OK;
}

int tc_split_attach_j(TcState &s, double unit_j, void *const *ops) {
  auto *p = static_cast<TcImpl *>(s.impl);
  p->unit_j = std::ldexp(unit_j, -(p->f16 ? 11 : 8) * (p->S - 1));
  int rc;
  for (int i = 0; i < 4; ++i)
    if ((rc = map_a(&p->maps.Jh[i / 2][i % 2], ops[i % 2], *p, p->Kh))) return rc;
  if ((rc = map_b(&p->maps.Jp, ops[2], *p, p->Kp))) return rc;
  s.tried_j = s.usable_j = true;
  return ATRIP_OK;
}

bool tc_sizes_ok(int No, int Nv, int64_t n_tuples, bool cplx) {
  // complex: the columns of both components of 8 levels fill TMEM at No = 32
  const double flops = (cplx ? 4.0 : 1.0) * (double)n_tuples * 12.0 * No * No * No * (No + Nv);
  // sums of the low levels are random: 5500 sqrt(6 K) for level 7, which stays
  // 8 standard deviations below the checked 2^22 up to K = 1400
  const int K = 2 * (Nv + No) * (cplx ? 2 : 1);
  return No >= 2 && (!cplx || No <= 32) && K <= 1400 && flops >= 1e9;
}

// Side of the (a,b,c) blocks tuples are processed in, 0 = list order.  In list
// order the ~150 tuples in flight read as many T_c slabs; where those exceed
// the L2 (129 MB, each die caching what it reads) blocks keep them resident;
// below it they gain nothing.  Two to four slices: side 4, in runs of 100 ms
// and more No=56/Nv=440 191 ms (6: 264, 8: 194), No=24/Nv=240 with 3 BF16
// slices 125 (list order 137, 6: 131), No=53/Nv=201 151 (6: 161).  The FP64
// form: side 6, No=24/Nv=240 11.8 ms (list order 12.5, 4: 13.0, 8: 12.3),
// No=40/Nv=300 62 (71, 77, 73); long runs at the power limit differ either
// way (No=24/Nv=240 6: 46 ms, 8: 42; No=37/Nv=151 list order 58, 6: 66).
int tc_tuple_block(int No, int Nv, int slices, int sm_count) {
  const double slab = 2.0 * slices * No * No * ((Nv + kKChunk - 1) / kKChunk * kKChunk);
  return slab * std::min(sm_count, Nv) > 64e6 ? (slices == kTcFp64Slices ? 6 : 4) : 0;
}

int tc_prepare(TcState &s, const DeviceTensors &dt, int No, int Nv, bool cplx, bool use_j,
               cudaStream_t st, int64_t *launches, bool *usable) {
  *usable = false;
  if (!s.tried) {
    const int rc = prepare_main(s, dt, No, Nv, cplx, st, launches);
    if (rc != ATRIP_OK || !s.usable) drop_impl(s);
    s.generation++;
    if (rc != ATRIP_OK) return rc;
    s.tried = true;
  }
  if (!s.usable) return ATRIP_OK;
  if (use_j && !s.tried_j) {
    const int rc = prepare_j(s, dt, st, launches);
    if (rc != ATRIP_OK || !s.usable_j) {
      auto *p = static_cast<TcImpl *>(s.impl);
      cudaFree(p->arena_j);
      p->arena_j = nullptr;
    }
    s.generation++;
    if (rc != ATRIP_OK) return rc;
    s.tried_j = true;
  }
  *usable = !use_j || s.usable_j;
  return ATRIP_OK;
}

void tc_buffers_free(TcBuffers &b) {
  cudaFreeHost(b.h_desc);
  cudaFree(b.d_desc);
  cudaFreeHost(b.h_prefix);
  cudaFree(b.d_prefix);
  cudaFree(b.planes);
  cudaFreeHost(b.h_flags);
  cudaFree(b.d_flags);
  cudaFree(b.d_queue);
  b = TcBuffers();
}

int tc_launch_prepare(const TcSystem *sys, int n, double tai_sign, int sm_count, TcBuffers &b,
                      int max_slots) {
  if (b.cap < n) {
    cudaFreeHost(b.h_desc);
    cudaFree(b.d_desc);
    cudaFreeHost(b.h_prefix);
    cudaFree(b.d_prefix);
    cudaFreeHost(b.h_flags);
    cudaFree(b.d_flags);
    b.h_desc = b.d_desc = nullptr;
    b.h_prefix = b.d_prefix = nullptr;
    b.h_flags = b.d_flags = nullptr;
    b.cap = 0;
    ATRIP_CUDA_TRY(cudaMallocHost(&b.h_desc, sizeof(TcDesc) * n));
    ATRIP_CUDA_TRY(device_alloc(&b.d_desc, sizeof(TcDesc) * n));
    ATRIP_CUDA_TRY(cudaMallocHost(&b.h_prefix, sizeof(int64_t) * (n + 1)));
    ATRIP_CUDA_TRY(device_alloc(&b.d_prefix, sizeof(int64_t) * (n + 1)));
    ATRIP_CUDA_TRY(cudaMallocHost(&b.h_flags, sizeof(int) * (n + 1)));
    ATRIP_CUDA_TRY(device_alloc(&b.d_flags, sizeof(int) * (n + 1)));
    b.cap = n;
  }
  if (!b.d_queue) ATRIP_CUDA_TRY(device_alloc(&b.d_queue, sizeof(unsigned long long)));
  auto *h = static_cast<TcDesc *>(b.h_desc);
  int P = 0, spp = 1, window = 0;
  const auto *p0 = static_cast<const TcImpl *>(n > 0 ? sys[0].state->impl : nullptr);
  const int S = p0 ? p0->S : kS;
  b.S = S;
  b.split = p0 && p0->split;
  b.f16 = p0 && p0->f16;
  b.lay_no = 0;
  b.lay_pass = 1;
  b.aslot = 0;
  b.nc = 1;
  b.pieces = 1;
  b.h_prefix[0] = 0;
  for (int k = 0; k < n; ++k) {
    const TcSystem &m = sys[k];
    auto *p = static_cast<TcImpl *>(m.state->impl);
    if (!p || !m.state->usable || (m.use_j && !m.state->usable_j) || p->S != S ||
        p->split != b.split || p->f16 != b.f16) {
      set_error("tensor-core FP64 form: operands not prepared");
      return ATRIP_ERR_STATE;
    }
    TcDesc d;
    std::memset(&d, 0, sizeof(d));
    d.maps = p->maps;
    d.epsi = m.dt->epsi;
    d.epsa = m.dt->epsa;
    d.tai = m.dt->tai;
    d.Vhh = m.dt->Vhh;
    d.tuples = m.tuples;
    d.triples = m.triples;
    d.tri_ef = m.tri_ef;
    d.e = m.e;
    d.ect = m.ect;
    d.unit = p->unit;
    d.unit_j = p->unit_j;
    d.tai_sign = tai_sign;
    d.t_begin = m.t_begin;
    d.No = m.No;
    d.Nv = m.Nv;
    d.P = p->P;
    d.rows = p->rows;
    d.spp = p->spp;
    d.n_triples = m.n_triples;
    d.use_j = m.use_j ? 1 : 0;
    b.pieces = std::max(b.pieces, m.use_j ? p->pieces_j : p->pieces);
    h[k] = d;
    P = std::max(P, p->P);
    b.nc = p->nc;  // the same for all: a batch holds real systems
    b.aslot = std::max(b.aslot, p->spp * p->rows * 128);
    spp = std::max(spp, p->spp);
    // an MMA reads 128 rows from its slice on, whatever the item's rows are
    window = std::max(window, (p->spp - 1) * p->rows * 128 + 128 * 128);
    b.lay_no = std::max(b.lay_no, m.No);
    if (m.use_j) b.lay_pass = 2;
    b.h_prefix[k + 1] = b.h_prefix[k] + std::max<int64_t>(0, m.t_end - m.t_begin);
  }
  b.n = n;
  b.total = b.h_prefix[n];
  b.grid = (int)std::min<int64_t>(b.total, sm_count);
  b.lay_cells = b.lay_no * b.lay_no * b.lay_no;
  // stack of 8 slices of P rows; an MMA's N, a multiple of 16, may read 8 rows more
  b.bslot = S * P * 128 + 1024;
  // rings: a K chunk takes S / spp A slots and one B slot, which must be free
  // by the time its first A slot is: chunk c's first slot is waited for until
  // the MMAs of the slot nslots before it are done, and the chunk nb before c
  // ends at or before that one if (nb - 1) chunks have nslots - 1 slots
  const int room = kSmemLimit - 1024 - kTailBytes;
  const int per_chunk = S / spp;  // of the system with the fewest A slots a chunk
  auto b_for = [&](int nslots) { return (nslots - 1 + per_chunk - 1) / per_chunk + 1; };
  // three slices and many orbitals: two slots, whose copies still cover the
  // MMAs of the other, leave 90 KB to L1 for the energy warps' gathers instead
  // of 24 (3 BF16 slices, 3 slots / 2: No=37 and Nv=60 56.1 / 47.5 ms, Nv=260 60.6
  // / 54.2, No=46/Nv=120 89 / 65, No=56/Nv=260 61 / 43; but No=36 43.8 / 43.9 and
  // 44.9 / 57.5, No=32 29.7 / 29.7 and 43.8 / 56.6)
  const int most = b.split && S == 3 && b.lay_no > 36 ? 2 : kMaxSlots;
  b.nslots = max_slots > 0 ? std::min(std::max(max_slots, 2), kMaxSlots) : most;
  while (b.nslots > 1 && b.nslots * b.aslot + b_for(b.nslots) * b.bslot > room) --b.nslots;
  b.nbslots = b_for(b.nslots);
  if (b.nslots * b.aslot + b.nbslots * b.bslot > room || b.nslots < 2) {
    set_error("tensor-core FP64 form: shared memory too small");
    return ATRIP_ERR_UNSUPPORTED;
  }
  // the last slot's window may reach past the B ring and the tail (few rows, a
  // shallow ring): it must still end in this block's shared memory
  const int end = b.nslots * b.aslot + b.nbslots * b.bslot + kTailBytes;
  b.smem = 1024 + (size_t)std::max(end, (b.nslots - 1) * b.aslot + window);
  const size_t cell = b.split ? 8 : 16;
  const size_t per_cta = (2 * 3 * cell + 8) * b.nc * b.lay_pass * b.lay_cells;
  const size_t need = per_cta * std::max(b.grid, 1);
  if (need > b.planes_bytes) {
    cudaFree(b.planes);
    b.planes = nullptr;
    b.planes_bytes = 0;
    ATRIP_CUDA_TRY(device_alloc(&b.planes, need));
    b.planes_bytes = need;
  }
  return ATRIP_OK;
}

int tc_launch_enqueue(const TcBuffers &b, const uint32_t *order, cudaStream_t st,
                      int64_t *launches) {
  ATRIP_CUDA_TRY(cudaMemcpyAsync(b.d_desc, b.h_desc, sizeof(TcDesc) * b.n, cudaMemcpyHostToDevice,
                                 st));
  ATRIP_CUDA_TRY(cudaMemcpyAsync(b.d_prefix, b.h_prefix, sizeof(int64_t) * (b.n + 1),
                                 cudaMemcpyHostToDevice, st));
  ATRIP_CUDA_TRY(cudaMemsetAsync(b.d_queue, 0, sizeof(unsigned long long), st));
  ATRIP_CUDA_TRY(cudaMemsetAsync(b.d_flags, 0, sizeof(int) * (b.n + 1), st));
  if (b.total == 0) return ATRIP_OK;
  TcArgs a;
  a.sys = static_cast<const TcDesc *>(b.d_desc);
  a.prefix = b.d_prefix;
  a.nsys = b.n;
  a.total = b.total;
  // several tuples a claim where every CTA has many (the tail stays even)
  a.claim = (int)std::max<int64_t>(1, std::min<int64_t>(8, b.total / (b.grid * 16ll)));
  a.order = order;
  a.queue = b.d_queue;
  a.flags = b.d_flags;
  a.planes = b.planes;
  a.wd = reinterpret_cast<double *>(static_cast<char *>(b.planes) +
                                    (size_t)b.grid * 2 * 3 * (b.split ? 8 : 16) * b.nc * b.lay_pass * b.lay_cells);
  a.lay_cells = b.lay_cells;
  a.lay_pass = b.lay_pass;
  a.nslots = b.nslots;
  a.nbslots = b.nbslots;
  a.aslot = b.aslot;
  a.bslot = b.bslot;
  a.unpublished = b.unpublished;
  auto kern = b.nc == 2 ? (b.pieces == 2 ? triples_tc_kernel<FmtZ<2>> : triples_tc_kernel<FmtZ<1>>)
                        : b.pieces == 2 ? triples_tc_kernel<FmtFp64<2>>
                                        : triples_tc_kernel<FmtFp64<1>>;
  if (b.split)
    kern = b.f16    ? triples_tc_kernel<Fmt<2, false, true, true>>
           : b.S == 2 ? triples_tc_kernel<Fmt<2, false, true, false>>
           : b.S == 3 ? triples_tc_kernel<Fmt<3, false, true, false>>
                      : triples_tc_kernel<Fmt<4, false, true, false>>;
  ATRIP_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      kSmemLimit));
  kern<<<b.grid, kThreads, b.smem, st>>>(a);
  ATRIP_CUDA_TRY(cudaGetLastError());
  *launches += 1;
  ATRIP_CUDA_TRY(cudaMemcpyAsync(b.h_flags, b.d_flags, sizeof(int) * (b.n + 1),
                                 cudaMemcpyDeviceToHost, st));
  return ATRIP_OK;
}

int tc_launch_check(const TcBuffers &b, TcState *const *states, bool *rerun) {
  *rerun = false;
  if (b.total == 0) return ATRIP_OK;
  if (b.h_flags[0] != 0) {
    set_error("tensor-core kernel: a bounded wait gave up (code " +
              std::to_string(b.h_flags[0]) + ")");
    return ATRIP_ERR_TIMEOUT;
  }
  for (int k = 0; k < b.n; ++k)
    if (b.h_flags[1 + k] != 0) {
      *rerun = true;
      drop_impl(*states[k]);
      states[k]->generation++;
    }
  return ATRIP_OK;
}

}  // namespace atrip_gb300
