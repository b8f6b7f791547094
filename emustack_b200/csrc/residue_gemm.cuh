// FP64-accurate complex GEMM on the INT8 tensor cores (tcgen05 kind::i8) by
// residue arithmetic.
//
//   C[r][s] = sum_k A[r][k] B[s][k]     complex, both operands K-major
//
// Each row of A and of B is scaled by a power of two and rounded to integers
// of 2-norm at most 2^62, so that every |Re C|, |Im C| <= ||a|| ||b|| <= 2^124
// (Cauchy-Schwarz), less than half the product 2^125.37 of 16 pairwise
// coprime moduli up to 256.  The integer product is then determined by its
// residues: one INT8 GEMM per modulus with exact INT32 accumulation, and the
// Chinese remainder theorem (128-bit integers) gives it back without any
// rounding; only the rounding of the operands to 62-bit rows and the final
// one to FP64 remain.  The method is K. Ozaki, T. Uchino and T. Imamura's
// "Ozaki scheme II" (2025) with row norms in place of row maxima.
//
// That rounding errs by up to 2^60.9 (rms) in the integers' unit, whatever the
// entry: FP64 sums err by some 2^-55.6 sum |a||b| (rms, K terms of random sign; more
// when they agree in sign).  Where sum |a||b| is far below ||a|| ||b|| (graded rows,
// localised fields, a diagonal operand) residues would therefore have fewer correct
// digits.  So a seventeenth product, of the operands' magnitudes in FP8 (e5m2: 2^-31
// of the row's norm is still there, and any non-zero value stays non-zero), gives
// sum |a||b| of each component to some 25 %, and a component below 2^-7 of its norms'
// largest product (kRgSafe) that is not exactly zero is left to FP64 sums: the 64 x 64
// tiles that hold one are computed again on the FP64 tensor cores, and the entries
// in question taken from there.  So no component has fewer digits than an FP64 sum
// gives, at any grading.  Of the GEMMs of interfaces and cascades with P = 634, M =
// 400, that is 2 % of the tiles of the triangular solves and none of the others',
// beside the products with a film's diagonal matrices (single products each).
//
// Why residues: the FP64 pipe of this chip delivers 36 TFLOP/s, its INT8 tensor
// cores two orders of magnitude more operations; a complex multiply-add costs
// 17 x 4 8-bit multiply-adds here.
//
// Complex products: planes (Ar, Ai) of A and (-Bi, Br, Bi) of B, so that
//   [Cr | Ci] = Ar [Br | Bi] + Ai [-Bi | Br]
// accumulates in one tensor-memory tile.
#pragma once
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "emu_cplx.cuh"
#include "emu_internal.h"

namespace emu {

constexpr int kRgMods = 16;
constexpr int kRgSlots = kRgMods + 1;  // the moduli's planes, then those of the magnitudes
constexpr int kRgBits = 62;            // row 2-norms are scaled to 2^61 .. 2^62
constexpr int kRgMagBits = 15;         // the magnitudes' to 2^14 .. 2^15 (e5m2 ends at 57 344)
constexpr float kRgSafe = 8388608.0f;  // 2^23: least sum |a||b| of a component, in the magnitudes' unit
constexpr int kRgPlanesA = 2, kRgPlanesB = 3;
constexpr int kRgTileM = 128, kRgTileN = 128, kRgStageK = 128;
// INT32 sums of 2 K products of magnitude <= 2^14 stay below 2^31, and the
// epilogue's 16-bit split below 2^22
constexpr int kRgMaxK = 61440;
constexpr int kRgMaxSplits = 16;

// ---- tables, computed at compile time
struct RgTab {
  int p[kRgMods];
  float invp[kRgMods];
  int c16[kRgMods];                  // 2^16 mod p, centred
  uint32_t clo[kRgMods], chi[kRgMods];  // 2^(8 j) mod p, centred, packed s8 x 4
  int init[kRgMods];                 // bits of the float V (see rg_residue), less 2^63 mod p
  // CRT weights as fractions of P, 80 bits: ((P / p)^-1 mod p) / p in a word of
  // 32, one of 32 and one of 16 bits
  uint32_t whi[kRgMods], wmid[kRgMods], wlo[kRgMods];
  uint64_t shi, smid, slo;           // their sums over the moduli
  double unit;                       // P / 2^64
};

constexpr int rg_centre(int r, int p) { return 2 * r > p ? r - p : r; }

constexpr RgTab rg_make_tab() {
  RgTab t{};
  const int mods[kRgMods] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193};
  unsigned __int128 P = 1;
  for (int i = 0; i < kRgMods; ++i) P *= (unsigned)mods[i];
  for (int i = 0; i < kRgMods; ++i) {
    const int p = mods[i];
    t.p[i] = p;
    t.invp[i] = 1.0f / (float)p;
    t.c16[i] = rg_centre((int)(65536 % p), p);
    int pw = 1 % p;
    uint32_t lo = 0, hi = 0;
    for (int j = 0; j < 8; ++j) {
      const uint32_t b = (uint32_t)(rg_centre(pw, p)) & 0xffu;
      if (j < 4) lo |= b << (8 * j);
      else hi |= b << (8 * (j - 4));
      pw = (int)((pw * 256) % p);
    }
    t.clo[i] = lo;
    t.chi[i] = hi;
    int b63 = 1;
    for (int j = 0; j < 63; ++j) b63 = (b63 * 2) % p;
    int neg = b63;  // the byte sum is at least -neg
    for (int j = 0, pj = 1 % p; j < 8; ++j, pj = (pj * 256) % p)
      if (rg_centre(pj, p) < 0) neg -= 255 * rg_centre(pj, p);
    const int V = (8388608 + neg + p - 1) / p * p;
    t.init[i] = 0x4B000000 + (V - 8388608) - b63;
    const unsigned __int128 Q = P / (unsigned)p;
    const int q = (int)(Q % (unsigned)p);
    int inv = 0;
    for (int x = 1; x < p; ++x)
      if ((q * x) % p == 1) inv = x;
    const unsigned __int128 W = (((unsigned __int128)(unsigned)inv << 81) / (unsigned)p + 1) >> 1;  // < 2^80
    t.whi[i] = (uint32_t)(W >> 48);
    t.wmid[i] = (uint32_t)(W >> 16);
    t.wlo[i] = (uint32_t)W & 0xffffu;
    t.shi += t.whi[i];
    t.smid += t.wmid[i];
    t.slo += t.wlo[i];
  }
  t.unit = (double)(uint64_t)(P >> 64) + (double)(uint64_t)P / 18446744073709551616.0;
  return t;
}
static_assert(rg_make_tab().unit > 0x1p61, "twice the largest product, 2^(2 x 62 + 1), is below the moduli's");

static __constant__ RgTab c_rg = rg_make_tab();  // for a modulus known at run time only

// one modulus as compile-time constants (immediate operands)
template <int I>
struct RgMod {
  static constexpr RgTab t = rg_make_tab();
  static constexpr int p = t.p[I], init = t.init[I];
  static constexpr uint32_t clo = t.clo[I], chi = t.chi[I];
  static constexpr uint32_t whi = t.whi[I], wmid = t.wmid[I], wlo = t.wlo[I];
};

// f(integral constant i) for i = 0 .. kRgMods - 1
template <int I>
struct RgIdx {
  static constexpr int value = I;
};
template <int I = 0, class F>
__device__ __forceinline__ void rg_for_mods(F &&f) {
  if constexpr (I < kRgMods) {
    f(RgIdx<I>{});
    rg_for_mods<I + 1>(f);
  }
}

// ---- operand rows
// Row scale from the largest |component| and the sum of squares of a row:
// the power of two 2^e with 2^61 <= ||x|| 2^e <= 2^62, returned as (2^e, 2^-e).  Rows
// outside the range where the scaled arithmetic is safe (non-finite values,
// magnitudes beyond 2^+-450, where squares leave FP64's range) return up = 0,
// down = -1: their products are FP64 sums.
struct RgScale {
  double up, down;
};

__device__ __forceinline__ double rg_pow2(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }

__device__ __forceinline__ RgScale rg_scale(double amax, double sumsq) {
  if (amax == 0.0 && sumsq == 0.0) return RgScale{1.0, 1.0};
  if (!(amax > 0x1p-450 && amax < 0x1p450 && sumsq < 0x1p930)) return RgScale{0.0, -1.0};
  // ||x|| < 2^x1 with x1 from the exponent of the sum of squares; one part
  // in 2^40 is added for the rounding of the sum
  const int ex = (int)((__double_as_longlong(sumsq * (1.0 + 0x1p-40)) >> 52) & 0x7ff) - 1022;  // sumsq < 2^ex
  const int x1 = (ex + 1) >> 1;  // 2^(2 x1) > sumsq
  const int e = kRgBits - x1;
  return RgScale{rg_pow2(e), rg_pow2(-e)};
}

// Centred residue of an integer, in the low byte.  v holds value + 2^63, so that
// all its bytes are unsigned.  dp4a adds sum_j byte_j (2^(8 j) mod p) - (2^63
// mod p) to the bit pattern of the float V, the smallest multiple of p that
// keeps the sum at or above 2^23, where a float's unit is 1.  Its quotient by
// p is rounded by adding 1.5 x 2^23 (one fused multiply-add), and the low byte
// of (sum - q p) is the residue: four operations for a modulus, and exactly
// centred (|r| <= (p - 1) / 2, checked for every reachable sum), so that a
// byte's negative is the negative's residue.  Modulus 256 is the low byte
// itself.
__device__ __forceinline__ int rg_dp4a(uint32_t a, uint32_t b, int c) {
  int d;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

template <int I>
__device__ __forceinline__ uint32_t rg_residue(uint64_t v) {
  if constexpr (I == 0) {
    static_assert(RgMod<0>::p == 256, "the first modulus is 256");
    return (uint32_t)v;
  } else {
    constexpr uint32_t clo = RgMod<I>::clo, chi = RgMod<I>::chi;
    constexpr int init = RgMod<I>::init, p = RgMod<I>::p;
    constexpr float ip = 1.0f / (float)p;
    const int d = rg_dp4a((uint32_t)v, clo, rg_dp4a((uint32_t)(v >> 32), chi, init));
    return (uint32_t)(d - __float_as_int(fmaf(__int_as_float(d), ip, 12582912.0f)) * p);
  }
}

__device__ __forceinline__ uint32_t rg_pack4(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
}

__device__ __forceinline__ uint64_t rg_int(double x, double up) {
  return (uint64_t)__double2ll_rn(x * up) + (1ull << 63);
}

// Writes the residues of 4 kW consecutive k of one operand row: planes are
// `plane` bytes apart, moduli kPlanes planes apart; `dst` points at this row's
// k in the first plane of the first modulus.
template <int kW>
struct RgVec;
template <>
struct RgVec<1> {
  using type = uint32_t;
};
template <>
struct RgVec<2> {
  using type = uint2;
};

// The magnitude of a value as e5m2, `um` = up 2^(kRgMagBits - kRgBits); what is not
// zero stays so.
__device__ __forceinline__ float rg_mag(double x, double um) {
  return x == 0.0 ? 0.0f : fmaxf((float)(fabs(x) * um), 0x1p-16f);
}
__device__ __forceinline__ uint32_t rg_mag4(float a, float b, float c, float d) {
  const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E5M2);
  const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, __NV_E5M2);
  return lo | hi << 16;
}

template <int kPlanes, int kW>
__device__ __forceinline__ void rg_store(const cd (&x)[4 * kW], double up, uint8_t *dst, long long plane) {
  using V = typename RgVec<kW>::type;
  {  // the magnitudes' planes, behind the moduli's
    uint8_t *at = dst + (long long)kRgMods * kPlanes * plane;
    uint32_t r[kW], m[kW];
    const double um = up * (1.0 / (double)(1ull << (kRgBits - kRgMagBits)));
#pragma unroll
    for (int h = 0; h < kW; ++h) {
      const cd *y = x + 4 * h;
      r[h] = rg_mag4(rg_mag(y[0].x, um), rg_mag(y[1].x, um), rg_mag(y[2].x, um), rg_mag(y[3].x, um));
      m[h] = rg_mag4(rg_mag(y[0].y, um), rg_mag(y[1].y, um), rg_mag(y[2].y, um), rg_mag(y[3].y, um));
    }
    if constexpr (kPlanes == 3) {
      *(V *)at = *(V *)m;
      at += plane;
    }
    *(V *)at = *(V *)r;
    *(V *)(at + plane) = *(V *)m;
  }
  uint64_t re[4 * kW], im[4 * kW];
#pragma unroll
  for (int j = 0; j < 4 * kW; ++j) {
    re[j] = rg_int(x[j].x, up);
    im[j] = rg_int(x[j].y, up);
  }
  rg_for_mods([&](auto i) {
    constexpr int I = decltype(i)::value;
    uint32_t r[kW], m[kW];
#pragma unroll
    for (int h = 0; h < kW; ++h) {
      r[h] = rg_pack4(rg_residue<I>(re[4 * h]), rg_residue<I>(re[4 * h + 1]), rg_residue<I>(re[4 * h + 2]),
                      rg_residue<I>(re[4 * h + 3]));
      m[h] = rg_pack4(rg_residue<I>(im[4 * h]), rg_residue<I>(im[4 * h + 1]), rg_residue<I>(im[4 * h + 2]),
                      rg_residue<I>(im[4 * h + 3]));
    }
    V *v = (V *)r, *w = (V *)m;
    if constexpr (kPlanes == 2) {
      *(V *)dst = *v;
      *(V *)(dst + plane) = *w;
    } else {
      uint32_t n[kW];
#pragma unroll
      for (int h = 0; h < kW; ++h) n[h] = __vneg4(m[h]);  // -128 (modulus 256) maps to itself
      *(V *)dst = *(V *)n;
      *(V *)(dst + plane) = *v;
      *(V *)(dst + 2 * plane) = *w;
    }
    dst += kPlanes * plane;
  });
}

// A component's sum of magnitudes as a byte: 0 if it is zero, else 5 bits of
// exponent and 3 of mantissa (rounded down) of values up to 2^31; below 1, 1.
__device__ __forceinline__ uint32_t rg_code(float s) {
  const int c = (int)(__float_as_uint(s) >> 20) - (127 << 3) + 1;
  return s > 0.0f ? (uint32_t)max(1, min(c, 255)) : 0u;
}
__device__ __forceinline__ float rg_uncode(uint32_t c) {
  return c > 1 ? __uint_as_float((c - 1 + (127u << 3)) << 20) : c ? 0x1p-20f : 0.0f;
}
__device__ __forceinline__ bool rg_unsafe(float s) { return s > 0.0f && s < kRgSafe; }

// The integer x whose residues, each plus `bias` (so that none is negative), are
// r(0) .. r(15): x / P is the sum of r_i w_i modulo 1, which 64-bit wrapping
// arithmetic does by itself, and |x| < P / 2 makes its signed reading the right
// one.  The weights are cut at 2^-80 and the sum rounded at 2^-64 of P, 2^61.4 (2^59.6
// rms), beside what rounding the operands' rows to 62 bits leaves (2^60.7 rms at
// most).  Residues may be sums over up to kRgMaxSplits K splits.
template <class R>
__device__ __forceinline__ double rg_crt(R &&r, uint32_t bias) {
  uint32_t hi = 0, lo = 0;  // lo < 16 x (255 kRgMaxSplits) x 2^16 < 2^32
  uint64_t mid = 0;
  rg_for_mods([&](auto i) {
    using W = RgMod<decltype(i)::value>;
    const uint32_t x = r(i);
    hi += x * W::whi;
    mid += (uint64_t)x * W::wmid;
    lo += x * W::wlo;
  });
  constexpr RgTab t = rg_make_tab();
  hi -= bias * (uint32_t)t.shi;
  const long long l = (long long)lo - (long long)(bias * t.slo);
  const uint64_t f = ((uint64_t)hi << 32) + mid - bias * t.smid + (uint64_t)((l + (1 << 15)) >> 16);
  return (double)(long long)f * t.unit;
}

// ---- the INT8 GEMMs (residue_gemm.cu)
struct RgPlan {
  int m, n, k;        // rows of A, rows of B, K
  int batch;
  int kp;             // row pitch of the residue planes (bytes): k rounded up to 128, so that no 128-byte box straddles lines
  int nt, ntiles, mtiles;
  int kper, nsplit;   // K per split (a multiple of 128)
  int ldn;            // row pitch of the result planes (bytes)
  long long bytesA, bytesB, bytesC;  // residue buffers of the whole batch
};

// Shapes and sizes for one batch of GEMMs; nsplit: K splits asked for (0: the
// rule's choice).  A split that gets no K still writes zeros.
RgPlan rg_plan(int m, int n, int k, int batch, int nsplit = 0);
// C [batch][split][slot][2][m][ldn] (signed bytes, in the last slot rg_code) from the
// operands' planes A [batch][slot][2][m][kp], B [batch][slot][3][n][kp], added to
// those in C if `add`; *err is set to 1 if a bounded wait gave up.
int rg_mma(const RgPlan &p, const uint8_t *A, const uint8_t *B, uint8_t *C, bool add, int *err, cudaStream_t s);

// ---- a whole GEMM of row-major FP64 matrices
// C = alpha A diag(dA) B + beta C for a batch (strides in elements; dA may be
// null).  C may not overlap A or B.
struct RgDense {
  int m, n, k, batch;
  cd alpha, beta;
  const cd *A;
  long long sA;
  int lda;
  const cd *B;
  long long sB;
  int ldb;
  cd *C;
  long long sC;
  int ldc;
  const cd *dA;
  long long sdA;
};

// Scratch for GEMMs of at most these sizes; more than one problem at a time
// and more rows of A at a time up to about 192 MB (96 MB, which stays in L2, took
// as long).
size_t rg_dense_scratch(int m, int n, int k, int batch);
// EMU_E_WORKSPACE if `bytes` holds not even 128 rows of one problem.
int rg_dense(const RgDense &g, void *ws, size_t bytes, cudaStream_t s);

}  // namespace emu
