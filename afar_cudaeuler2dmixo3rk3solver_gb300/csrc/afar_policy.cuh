// Precision policies and small math helpers shared by the AFAR kernels.
//
// A policy fixes the arithmetic type of each part of the stage:
//   W   stored primitive state (cells and ghosts)
//   S   staged stencil values, limiter arithmetic, least-squares and O3 weights
//   G   gradients, face values, TVD states, central flux
//   D   Riemann dissipation (Roe / KFVS)
//   RC  R and Cv as seen by the dissipation
//   F   stored face flux
// The conserved state, the residual gather and the RK update are FP64 under every policy.
//
// PolicyRef reproduces the reference's own mix (float stencils/weights/limiters/dissipation,
// double elsewhere; reference cudaLimiter.h:83-98, basicDataStructure.h:67-73,134,150,
// cudaRiemannSolver.h:16-136).  Under it every expression below is written with the same operand
// types and order as the reference kernel it restates, so nvcc makes the same rounding and
// FMA-contraction decisions; that is what makes the 1e-12 / identical-switch parity possible.
#pragma once

#include <cuda.h>  // CUtensorMap (the type only: the library does not link the driver API)
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

namespace afar {

struct PolicyRef {
  static constexpr int id = 0;
  using W = double;
  using S = float;
  using G = double;
  using D = float;
  using RC = double;
  using F = double;
  static constexpr bool exact_blend = true;
};

struct PolicyFP64 {
  static constexpr int id = 1;
  using W = double;
  using S = double;
  using G = double;
  using D = double;
  using RC = double;
  using F = double;
  static constexpr bool exact_blend = false;
};

struct PolicyMixed {
  static constexpr int id = 2;
  using W = float;
  using S = float;
  using G = float;
  using D = float;
  using RC = float;
  using F = float;
  static constexpr bool exact_blend = false;
};

template <class T>
struct alignas(4 * sizeof(T)) V4 {
  T x, y, z, w;
};
template <class T>
struct alignas(2 * sizeof(T)) V2 {
  T x, y;
};

// A literal of type T that equals the reference's float literal when T is float (x##f) and the
// double literal otherwise.
#define AFAR_LIT(T, x) (std::is_same<T, float>::value ? (T)(x##f) : (T)(x))

// Overloads that resolve like the CUDA C++ math overloads the reference calls.
__device__ __forceinline__ float fmx(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ double fmx(double a, double b) { return fmax(a, b); }
__device__ __forceinline__ float fmn(float a, float b) { return fminf(a, b); }
__device__ __forceinline__ double fmn(double a, double b) { return fmin(a, b); }
__device__ __forceinline__ float fab(float a) { return fabsf(a); }
__device__ __forceinline__ double fab(double a) { return fabs(a); }
__device__ __forceinline__ float sqr_(float a) { return sqrtf(a); }
__device__ __forceinline__ double sqr_(double a) { return sqrt(a); }
__device__ __forceinline__ float rsq_(float a) { return rsqrtf(a); }
__device__ __forceinline__ double rsq_(double a) { return rsqrt(a); }
__device__ __forceinline__ float erfc_(float a) { return erfcf(a); }
__device__ __forceinline__ double erfc_(double a) { return erfc(a); }
__device__ __forceinline__ float exp_(float a) { return expf(a); }
__device__ __forceinline__ double exp_(double a) { return exp(a); }

// ---------------------------------------------------------------- sparing the FP64 pipe
// GB300 issues two FP64 lanes a clock and SM: one FP64 warp instruction takes the pipe 16 clocks, in
// which the four schedulers issue 64 others.  Comparisons, minima, conversions and the compiler's
// division and root sequences all run on that pipe, so the fp64 policy compares doubles as integers,
// and starts reciprocals from the FP32 approximation, refined by one third-order step in FP64.
__device__ __forceinline__ unsigned long long dbits(const double x) {
  return (unsigned long long)__double_as_longlong(x);
}
constexpr unsigned long long kInfBits = 0x7FF0000000000000ull;
// by the high word: as a mask on all 64 bits the compiler makes it an addition on the FP64 pipe
__device__ __forceinline__ double dabs_(const double x) {
  return __hiloint2double(__double2hiint(x) & 0x7FFFFFFF, __double2loint(x));
}
// by the high word alone (every NaN that arithmetic produces has a high fraction bit set): as a test
// on all 64 bits the compiler makes it a comparison on the FP64 pipe
__device__ __forceinline__ bool dnan_(const double x) { return (__double2hiint(x) & 0x7FFFFFFF) > 0x7FF00000; }
// |x| < c and |x| >= c for a constant c > 0; false on NaN, as the comparisons are.
__device__ __forceinline__ bool abs_lt(const double x, const double c) { return dbits(dabs_(x)) < dbits(c); }
__device__ __forceinline__ bool abs_ge(const double x, const double c) {
  return dbits(dabs_(x)) - dbits(c) <= kInfBits - dbits(c);
}
__device__ __forceinline__ bool abs_lt(const float x, const float c) { return fabsf(x) < c; }
__device__ __forceinline__ bool abs_ge(const float x, const float c) { return fabsf(x) >= c; }
__device__ __forceinline__ bool gt_zero(const double x) { return dbits(x) - 1ull < kInfBits; }
__device__ __forceinline__ bool le_zero(const double x) {
  return dbits(x) == 0ull || dbits(x) - 0x8000000000000000ull <= kInfBits;
}
__device__ __forceinline__ double flip_sign(const double x, const int bit) {
  return __hiloint2double(__double2hiint(x) ^ bit, __double2loint(x));
}
// positive, normal and finite, by the high word
__device__ __forceinline__ bool pos_normal(const double x) {
  return (unsigned)__double2hiint(x) - 0x00100000u < 0x7FE00000u;
}
__device__ __forceinline__ bool neg_(const double x) { return (long long)dbits(x) < 0; }  // the sign bit
// fmin of two doubles without a sign (NaN loses, as in fmin)
__device__ __forceinline__ double min_nonneg(const double a, const double b) { return dbits(b) < dbits(a) ? b : a; }
// fmax and fmin for any operands (of two zeros either; NaN loses): the bits of a double, its lower 63
// flipped where it is negative, order like the numbers.
__device__ __forceinline__ long long dkey(const double x) {
  const long long b = __double_as_longlong(x);
  return b ^ ((b >> 63) & 0x7FFFFFFFFFFFFFFFll);
}
__device__ __forceinline__ double dmax_(const double a, const double b) {
  return dnan_(a) || (dkey(b) > dkey(a) && !dnan_(b)) ? b : a;
}
__device__ __forceinline__ double dmin_(const double a, const double b) {
  return dnan_(a) || (dkey(b) < dkey(a) && !dnan_(b)) ? b : a;
}
// the policy's larger and smaller of two: fmaxf, fminf, or the integer forms
__device__ __forceinline__ float gmx(const float a, const float b) { return fmaxf(a, b); }
__device__ __forceinline__ float gmn(const float a, const float b) { return fminf(a, b); }
__device__ __forceinline__ double gmx(const double a, const double b) { return dmax_(a, b); }
__device__ __forceinline__ double gmn(const double a, const double b) { return dmin_(a, b); }
// x as a float to 20 bits from its high word (zero below the range of float), for estimates
__device__ __forceinline__ float top_float(const double x) {
  const int hi = __double2hiint(x), a = hi & 0x7FFFFFFF;
  const unsigned m = a < 0x38100000 ? 0u : a >= 0x47F00000 ? 0x7F800000u : (unsigned)(a - 0x38000000) << 3;
  return __uint_as_float(m | ((unsigned)hi & 0x80000000u));
}
// 1/x: y0 to 23 bits from the mantissa's FP32 reciprocal, then y0 (1 + e + e^2) with e = 1 - x y0,
// whose remainder e^3 is below 2^-66: three FP64 operations, within an ulp.  Zeros, subnormals,
// infinities, NaN and reciprocals that are subnormal take the division.
__device__ __forceinline__ double rcp64(const double x) {
  const int hi = __double2hiint(x), lo = __double2loint(x);
  const int e = (hi >> 20) & 0x7FF;
  if ((unsigned)(e - 1) > 2042u) return 1.0 / x;
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__int_as_float(0x3F800000 | ((hi & 0xFFFFF) << 3) | ((unsigned)lo >> 29))));
  const int rb = __float_as_int(r);
  const double y0 = __hiloint2double(((rb >> 3) + (896 + 1023 - e) * (1 << 20)) | (hi & (int)0x80000000), rb << 29);
  const double d = __fma_rn(-x, y0, 1.0);
  return __fma_rn(y0, __fma_rn(d, d, d), y0);
}
// 1/sqrt(x): y0 the same way from x scaled by an even power of two into [1, 4), then
// y0 (1 + e/2 + 3/8 e^2) with e = 1 - x y0^2 (Halley's step): five FP64 operations.
__device__ __forceinline__ double rsq64(const double x) {
  const int hi = __double2hiint(x), lo = __double2loint(x);
  const int e = hi >> 20;  // the sign bit makes it negative
  if ((unsigned)(e - 1) > 2045u) return rsqrt(x);
  const int k = (e - 1023) >> 1;
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__int_as_float(((e - 896 - 2 * k) << 23) | ((hi & 0xFFFFF) << 3) | ((unsigned)lo >> 29))));
  const int rb = __float_as_int(r);
  const double y0 = __hiloint2double((rb >> 3) + ((896 - k) << 20), rb << 29);
  const double d = __fma_rn(-__dmul_rn(x, y0), y0, 1.0);
  return __fma_rn(__dmul_rn(y0, d), __fma_rn(0.375, d, 0.5), y0);
}

// float to double and double to float (to nearest, ties to even) on integers: as conversions they take
// the FP64 pipe.  Whatever is not a normal float or zero on the float's side takes the conversion.
__device__ __forceinline__ double to_double(const float x) {
  const unsigned b = __float_as_uint(x), m = b & 0x7FFFFFFFu;
  if (m - 0x00800000u < 0x7F000000u || m == 0u)
    return __hiloint2double((int)((b & 0x80000000u) | (m ? (m >> 3) + 0x38000000u : 0u)), (int)(m << 29));
  double y;
  asm volatile("cvt.f64.f32 %0, %1;" : "=d"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float to_float(const double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x), m = hi & 0x7FFFFFFFu;
  if (m - 0x38100000u < 0x47EFFFFFu - 0x38100000u || (m | lo) == 0u) {  // below the largest float
    const unsigned t = m ? __funnelshift_l(lo, m - 0x38000000u, 3) : 0u;
    const unsigned up = ((lo & 0x1FFFFFFFu) + 0x0FFFFFFFu + (t & 1u)) >> 29;
    return __uint_as_float((hi & 0x80000000u) | (t + up));
  }
  float y;
  asm volatile("cvt.rn.f32.f64 %0, %1;" : "=f"(y) : "d"(x));
  return y;
}
// a/b rounded to nearest from r = rcp64(b): q = a r is within two ulp, its remainder a - b q comes out of
// the fused multiply-add and corrects it (Markstein 1990) to 2^-103 before the last rounding.  Operands
// far from the ends of the range, or a = 0; others take the division.
__device__ __forceinline__ bool div64_range(const double x) {
  return ((unsigned)__double2hiint(x) & 0x7FFFFFFFu) - 0x26F00000u < 0x32000000u;  // 2^-400 to 2^400
}
__device__ __forceinline__ double div64(const double a, const double b, const double r) {
  const bool zero = (dbits(a) << 1) == 0ull;
  if (!div64_range(b) || !(zero || div64_range(a))) return a / b;
  const double q = __dmul_rn(a, r);
  const double c = __fma_rn(__fma_rn(-b, q, a), r, q);
  return zero ? q : c;  // (a zero keeps its sign)
}
__device__ __forceinline__ double div64(const double a, const double b) { return div64(a, b, rcp64(b)); }
// x/2 by the exponent
__device__ __forceinline__ double half64(const double x) {
  const int hi = __double2hiint(x);
  if ((((unsigned)hi & 0x7FFFFFFFu) - 0x00200000u) < 0x7FC00000u) return __hiloint2double(hi - 0x00100000, __double2loint(x));
  double y;  // zeros, subnormals, halves that are, and what is not finite
  asm volatile("mul.rn.f64 %0, %1, 0d3FE0000000000000;" : "=d"(y) : "d"(x));
  return y;
}
// c1*a + c2*b of two conditions, one true: the chosen one, as the sum leaves it (a negative zero stays
// one only next to a negative operand); anything not finite takes the sum.
static __device__ __noinline__ double blend64_sum(const bool c1, const bool c2, const double a, const double b) {
  return __dadd_rn(__dmul_rn((double)c1, a), __dmul_rn((double)c2, b));
}
__device__ __forceinline__ double blend64(const bool c1, const bool c2, const double a, const double b) {
  const unsigned ha = (unsigned)__double2hiint(a), hb = (unsigned)__double2hiint(b);
  if (c1 == c2 || (ha & 0x7FF00000u) == 0x7FF00000u || (hb & 0x7FF00000u) == 0x7FF00000u)
    return blend64_sum(c1, c2, a, b);
  unsigned hi = c1 ? ha : hb;
  const unsigned lo = (unsigned)(c1 ? __double2loint(a) : __double2loint(b)), other = c1 ? hb : ha;
  if (hi == 0x80000000u && lo == 0u) hi &= other;
  return __hiloint2double((int)hi, (int)lo);
}

// Programmatic dependent launch: a kernel that says pdl_next() in every block lets the one after it on
// the stream start, whose pdl_wait() returns when the first is complete and its writes are visible.
// Neither does anything in a launch without that attribute.
template <bool EARLY = true>
__device__ __forceinline__ void pdl_next() {
  if constexpr (EARLY) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <bool EARLY = true>
__device__ __forceinline__ void pdl_wait() {
  if constexpr (EARLY) asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Bulk global->shared copies (cp.async.bulk, the TMA unit's untiled form) completing on an
// mbarrier.  Both addresses 16-byte aligned, size a multiple of 16.
__device__ __forceinline__ unsigned smem_addr(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(bytes)
               : "memory");
}
// Counts `bytes` as arrived without a copy (test hooks).
__device__ __forceinline__ void mbar_complete_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.complete_tx.relaxed.cta.shared::cta.b64 [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_to_smem(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                   smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Waits for phase `parity` of the barrier for at most `limit` SM clocks (by default 2^31, about
// 1 s); false if it gave up.
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long* bar, unsigned parity,
                                                  const long long limit = 1ll << 31) {
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity))
    if (clock64() - t0 > limit) return false;
  return true;
}

// cond ? a : b.  The reference writes these selections as arithmetic blends
// (c1*a + c2*b with c1, c2 in {0,1}); the ref policy keeps the blend so that signed zeros and
// non-finite operands propagate the same way.
template <class P, class A, class B>
__device__ __forceinline__ auto pick(bool c1, bool c2, A a, B b) -> decltype(a * 1 + b * 1) {
  if constexpr (P::exact_blend) {
    return c1 * a + c2 * b;
  } else {
    using R = decltype(a * 1 + b * 1);
    return c1 ? (R)a : (R)b;
  }
}

// ---------------------------------------------------------------- float-pair ("double-float") values
// A value hi + lo with |lo| <= ulp(hi)/2 (about 48 significant bits) built from FP32 operations
// only, for the mixed policy's conserved state: GB300's FP64 pipe runs at 1/53 of FP32.  The
// error-free transformations are Knuth's two-sum, Dekker's fast two-sum (|a| >= |b|) and the
// FMA two-product; the explicitly rounded __fadd_rn/__fmul_rn keep the compiler from fusing a
// product into a later sum, which would break the transformations.
struct DF {
  float hi, lo;
};
// The conserved state of one cell as float pairs: 32 bytes, like V4<double>.
struct alignas(16) DF4 {
  V4<float> hi, lo;
};

__device__ __forceinline__ DF df_two_sum(const float a, const float b) {
  const float s = __fadd_rn(a, b);
  const float bp = __fadd_rn(s, -a);
  return DF{s, __fadd_rn(__fadd_rn(a, -__fadd_rn(s, -bp)), __fadd_rn(b, -bp))};
}
__device__ __forceinline__ DF df_fast_two_sum(const float a, const float b) {
  const float s = __fadd_rn(a, b);
  return DF{s, __fadd_rn(b, -__fadd_rn(s, -a))};
}
// a + b, both float pairs (the accurate sum: two-sums of both parts).
__device__ __forceinline__ DF df_add(const DF a, const DF b) {
  DF s = df_two_sum(a.hi, b.hi);
  const DF t = df_two_sum(a.lo, b.lo);
  s = df_fast_two_sum(s.hi, __fadd_rn(s.lo, t.hi));
  return df_fast_two_sum(s.hi, __fadd_rn(s.lo, t.lo));
}
// a + b, b a float.
__device__ __forceinline__ DF df_add(const DF a, const float b) {
  const DF s = df_two_sum(a.hi, b);
  return df_fast_two_sum(s.hi, __fadd_rn(s.lo, a.lo));
}
// a * b.
__device__ __forceinline__ DF df_mul(const DF a, const DF b) {
  const float p = __fmul_rn(a.hi, b.hi);
  float e = __fmaf_rn(a.hi, b.hi, -p);
  e = __fmaf_rn(a.hi, b.lo, e);
  e = __fmaf_rn(a.lo, b.hi, e);
  return df_fast_two_sum(p, e);
}
// a * a.
__device__ __forceinline__ DF df_sqr(const DF a) {
  const float p = __fmul_rn(a.hi, a.hi);
  const float e = __fmaf_rn(__fmul_rn(2.f, a.hi), a.lo, __fmaf_rn(a.hi, a.hi, -p));
  return df_fast_two_sum(p, e);
}
// a / b given r ~ 1/b.hi: one correction of the float quotient, q = q0 + (a - q0 b) r.
__device__ __forceinline__ DF df_div(const DF a, const DF b, const float r) {
  const float q0 = __fmul_rn(a.hi, r);
  const DF qb = df_mul(DF{q0, 0.f}, b);
  const DF rem = df_add(a, DF{-qb.hi, -qb.lo});
  return df_fast_two_sum(q0, __fmul_rn(__fadd_rn(rem.hi, rem.lo), r));
}

}  // namespace afar
