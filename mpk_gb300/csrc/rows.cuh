// Row arithmetic and flag waits shared by the kernels (device code).
#ifndef MPKG_ROWS_CUH
#define MPKG_ROWS_CUH

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "../../include/mpk_gb300.h"
#include "host.h"

namespace {

constexpr int kErrTimeout = 2;
constexpr int kErrBounds = 3;
constexpr long kSpinLimit = 4000000;  // polls of one flag (~1 s with backoff)

#define CUDA_TRY(expr)                                                             \
  do {                                                                             \
    cudaError_t e_ = (expr);                                                       \
    if (e_ != cudaSuccess)                                                         \
      return fail(kECuda, std::string(#expr) + ": " + cudaGetErrorString(e_));     \
  } while (0)

template <int ARITH>
__device__ __forceinline__ double row_term(double s, double a, double x) {
  if (ARITH == MPKG_ARITH_SEPARATE) return __dadd_rn(s, __dmul_rn(a, x));
  return __fma_rn(a, x, s);
}

// a * x rounded to nearest even on the integer pipes: the 53 x 53 bit product
// as four 32-bit multiplies, the top 53 bits rounded on what lies below.
// False (and no result) unless both exponents are within 2^-503 .. 2^496,
// where neither operand nor product is subnormal, zero, infinite or NaN.
// GB300 has two FP64 lanes per SM and clock, so an FP64 product holds its
// scheduler's pipe for 64 cycles; this one takes about 40 issue slots of the
// idle integer pipes beside it.  Products per second, 1024 threads per SM:
// 0.50 T all FP64, 0.53 T all integer, 0.98 T half and half.
__device__ __forceinline__ bool mul_int(double a, double x, double *p) {
  const unsigned long long A = (unsigned long long)__double_as_longlong(a);
  const unsigned long long X = (unsigned long long)__double_as_longlong(x);
  const uint32_t ea = (uint32_t)(A >> 52) & 0x7FFu, ex = (uint32_t)(X >> 52) & 0x7FFu;
  if (ea - 520u >= 1000u || ex - 520u >= 1000u) return false;
  const unsigned long long ma = (A << 11) | 0x8000000000000000ull;                     // top bit 63
  const unsigned long long mx = (X & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;        // top bit 52
  const uint32_t al = (uint32_t)ma, ah = (uint32_t)(ma >> 32), xl = (uint32_t)mx, xh = (uint32_t)(mx >> 32);
  const unsigned long long t0 = (unsigned long long)al * xl;
  const unsigned long long t1 = (unsigned long long)ah * xl + (t0 >> 32);
  const unsigned long long t2 = (unsigned long long)al * xh + (uint32_t)t1;
  const unsigned long long t3 = (unsigned long long)ah * xh + (t1 >> 32);
  unsigned long long hi = t3 + (t2 >> 32), lo = (t2 << 32) | (uint32_t)t0;             // hi: 52 or 53 bits
  const uint32_t n = ((uint32_t)(hi >> 52) & 1u) ^ 1u;
  hi = (hi << n) | ((lo >> 63) & n);
  lo <<= n;  // its low 11 bits are zero: no overflow below
  hi += lo + 0x7FFFFFFFFFFFFFFFull + (hi & 1ull) < lo ? 1ull : 0ull;
  // hi's bit 52 (53 after a carry) adds to the exponent field
  *p = __longlong_as_double((long long)(((A ^ X) & 0x8000000000000000ull) |
                                        (((unsigned long long)(ea + ex - 1023u - n) << 52) + hi)));
  return true;
}

// row_term(+0, a, x): the first term of a row is a product alone.
template <int ARITH>
__device__ __forceinline__ double row_first(double a, double x) {
  double p;
  return mul_int(a, x, &p) ? p : row_term<ARITH>(0.0, a, x);
}

// row_term with the separately rounded product on the integer pipes.
template <int ARITH>
__device__ __forceinline__ double row_next(double s, double a, double x) {
  double p;
  if (ARITH == MPKG_ARITH_SEPARATE) return __dadd_rn(s, mul_int(a, x, &p) ? p : __dmul_rn(a, x));
  return row_term<ARITH>(s, a, x);
}

__device__ __forceinline__ unsigned int ld_acquire(const unsigned int *p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void st_release(unsigned int *p, unsigned int v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// ------------------------------------------------------------------------
// Double-float ("df64") arithmetic on the FP32 pipes.  A value is an
// unevaluated sum h + l of two floats with |l| <= ulp(h)/2 after
// normalisation (48 significand bits).  Products use the exact FMA
// residual; sums use Knuth's TwoSum.  Intrinsics (__fmul_rn, __fadd_rn)
// keep the compiler from contracting the error-free transformations.
// FP64 <-> df64 conversions use integer bit manipulation so that they do
// not occupy the narrow FP64 pipe.
// ------------------------------------------------------------------------
__device__ __forceinline__ float2 df_split(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int e = (int)((b >> 52) & 0x7FF);
  const int E = e - 1023;
  const unsigned int sgn = (unsigned int)(b >> 63) << 31;
  if (e == 0x7FF || E > 127) {  // inf/nan or beyond the float range
    const float h = __double2float_rn(x);
    return make_float2(h, 0.0f);
  }
  if (E < -126) return make_float2(0.0f, 0.0f);  // below the df64 range
  const unsigned long long m = b & 0xFFFFFFFFFFFFFull;
  const float h = __uint_as_float(sgn | ((unsigned)(E + 127) << 23) | (unsigned)(m >> 29));
  const unsigned int rem = (unsigned int)(m & 0x1FFFFFFFull);  // low 29 bits, weight 2^(E-52)
  float lo = 0.0f;
  if (rem != 0 && E - 52 >= -126) {
    lo = __fmul_rn(__uint2float_rn(rem), __uint_as_float((unsigned)(E - 52 + 127) << 23));
    lo = __uint_as_float(__float_as_uint(lo) | sgn);
  }
  return make_float2(h, lo);
}

__device__ __forceinline__ double df_widen(float f) {
  const unsigned int u = __float_as_uint(f);
  const unsigned int e = (u >> 23) & 0xFF;
  if (e == 0) return __longlong_as_double((long long)((unsigned long long)(u >> 31) << 63));  // +-0
  if (e == 0xFF) return (double)f;
  return __longlong_as_double((long long)(((unsigned long long)(u >> 31) << 63) |
                                          ((unsigned long long)(e + 896) << 52) |
                                          ((unsigned long long)(u & 0x7FFFFF) << 29)));
}

__device__ __forceinline__ double df_to_double(float2 v) { return __dadd_rn(df_widen(v.x), df_widen(v.y)); }

// s += a * x in double-float
__device__ __forceinline__ void df_mac(float2 a, float2 x, float &sh, float &sl) {
  const float p = __fmul_rn(a.x, x.x);
  float e = __fmaf_rn(a.x, x.x, -p);
  e = __fmaf_rn(a.x, x.y, e);
  e = __fmaf_rn(a.y, x.x, e);
  const float s = __fadd_rn(sh, p);
  const float bp = __fadd_rn(s, -sh);
  const float t = __fadd_rn(__fadd_rn(sh, -__fadd_rn(s, -bp)), __fadd_rn(p, -bp));
  sh = s;
  sl = __fadd_rn(sl, __fadd_rn(t, e));
}

__device__ __forceinline__ float2 df_norm(float sh, float sl) {
  const float h = __fadd_rn(sh, sl);
  const float l = __fadd_rn(sl, -__fadd_rn(h, -sh));
  return make_float2(h, l);
}

// s += x in double-float (two-sum of the high parts, low parts added)
__device__ __forceinline__ void df_acc(float2 x, float &sh, float &sl) {
  const float s = __fadd_rn(sh, x.x);
  const float bp = __fadd_rn(s, -sh);
  const float t = __fadd_rn(__fadd_rn(sh, -__fadd_rn(s, -bp)), __fadd_rn(x.x, -bp));
  sh = s;
  sl = __fadd_rn(sl, __fadd_rn(t, x.y));
}

// a * v in double-float (v normalised)
__device__ __forceinline__ float2 df_scale(float2 a, float2 v) {
  const float p = __fmul_rn(a.x, v.x);
  float e = __fmaf_rn(a.x, v.x, -p);
  e = __fmaf_rn(a.x, v.y, e);
  e = __fmaf_rn(a.y, v.x, e);
  return df_norm(p, e);
}

__device__ __forceinline__ float to_f32(float v) { return v; }
__device__ __forceinline__ float to_f32(__nv_bfloat16 v) { return __bfloat162float(v); }

// Separate arithmetic: the first kIntTerms terms of a row have integer
// products, the others FP64 ones (110 x 111 x 112, 1/deg, 8 levels, all on the
// FP64 pipe 392 us; 4, 5, 6, 7 of 7: 273, 255, 252, 258).
constexpr int kIntTerms = 6;

// ---- 1-D bulk copies (TMA) into shared memory ----
__device__ __forceinline__ unsigned smem_u32(const void *p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned long long *bar) {
  asm volatile("mbarrier.init.shared.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned long long *bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned long long *bar, unsigned phase) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok) : "r"(smem_u32(bar)), "r"(phase) : "memory");
  return ok != 0;
}
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, unsigned bytes, unsigned long long *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ bool tr_wait(unsigned long long *bar, unsigned phase, int *err) {
  long spins = 0;
  while (!mbar_try(bar, phase)) {
    if (spins > 16) __nanosleep(64);
    if (++spins > kSpinLimit) {  // a copy of this CTA never completed: report, drain with a second bound
      if (threadIdx.x == 0) atomicCAS(err, 0, kErrTimeout);
      for (long s2 = 0; s2 < kSpinLimit && !mbar_try(bar, phase); s2++) __nanosleep(256);
      return false;
    }
  }
  return true;
}

}  // namespace

#endif
