// math_fast64.cuh -- the FP64 kernels' arithmetic: the same bits as pmp_math.h
// and IEEE division, arranged for the GPU.
//
// MathPlain evaluates pmp_math.h and `/` as they stand.  MathFast returns the
// same values for ordinary arguments without a branch: an argument that
// pmp_math.h sends down a rare path, or a divisor whose exponent is not in the
// middle of the range, sets `odd`, and the caller then evaluates the whole
// droplet sub-cycle again with MathPlain (redo_subcycle).
// Dividends are not checked.  A quotient has the bits of IEEE division when the
// dividend's magnitude is within 2^+-600, and a zero dividend gives +0 (-0 too).
// Of a smaller dividend the last bits can differ (a - b q is rounded), of a
// larger or infinite one the quotient can be NaN.  The droplets' bits do not
// depend on it: an infinite or NaN gas state reaches a checked divisor (the
// mixture's weight, the pressure) or check_finite (the Reynolds number), a
// droplet's temperature, diameter and fractions reach the density's reciprocal
// or a logarithm, and a tiny mass fraction is a term of sums of ordinary ones.
// Why: each branch ends a basic block, so that in the plain form every
// exponential, logarithm and division of the droplet physics ran its
// dependent chain alone (57 elementary functions and 60 divisions per
// sub-cycle, 7300 instructions a droplet of which 34 % FP64; the warps waited
// 3.3 cycles per issue on fixed latencies).  Measured, update kernel of 2M
// two-fuel droplets, 4 sub-cycles: 3.48 -> 2.15 ms (5200 instructions, 41 %
// FP64); 100k one-fuel droplets 81 -> 36 us; 800 droplets (the latency of one)
// 29 -> 14 us.  Species loops left rolled (mass fractions in shared memory,
// code 8 % smaller) measured 4 % slower.
//  - exp: k from the low word of x / (ln2/128) + 1.5 2^52 (the sum rounds to
//    the nearest integer, ties to even, as rint does), 2^m added to the
//    exponent field (the result is normal); no conversion
//    instructions, which run at a quarter of the FP64 rate.
//  - log: table index from the low word of fma_rz(|m - 1|, 128, 1.5 2^52)
//    (truncation), the exponent as a double by an exact subtraction.
//  - tables in shared memory (3.3 KB a CTA): a warp's 32 table reads touch up
//    to 8 lines of L1.
//  - a / b from a reciprocal y of b by q = RN(a y), r = RN(a - b q),
//    RN(q + r y): correctly rounded once y is 1/b correctly rounded
//    (Markstein, IBM J. Res. Dev. 34(1), 1990; Brisebarre, Muller and Raina,
//    IEEE Trans. Comput. 53(8), 2004).  A divisor that is a launch constant
//    brings y from the host, one that divides several numbers forms it once.
//    1/b itself: Newton steps from the hardware estimate, the last one
//    rounding correctly unless b's significand is all ones (Markstein), where
//    1/b is known.
// tests/test_gpu_math.py compares every function with the plain one, bit for
// bit, and droplets with rare dividends with the oracle.
#pragma once

#include "pmp_math.h"

namespace pmp {

struct MathTables {
  double2 loga[PMP_LOG_NTAB];  // {1/c, hi of -log(1/c)}
  double logl[PMP_LOG_NTAB];   // lo
  double exp2[PMP_EXP_N];
};

// the CTA's tables; stage_math_tables before the first use, and a barrier
__device__ __forceinline__ MathTables& math_tables()
{
  __shared__ MathTables t;
  return t;
}

__device__ __forceinline__ void stage_math_tables()
{
  MathTables& t = math_tables();
  for (int i = threadIdx.x; i < PMP_EXP_N; i += blockDim.x) {
    t.exp2[i] = pmp_dev_exp2[i];
    if (i < PMP_LOG_NTAB) {
      t.loga[i] = make_double2(pmp_dev_loginv[i], pmp_dev_loglhi[i]);
      t.logl[i] = pmp_dev_logllo[i];
    }
  }
  static_assert(PMP_LOG_NTAB <= PMP_EXP_N, "one loop");
}

// a divisor and, in MathFast, its reciprocal
struct Divisor {
  double b, y;
};

struct MathPlain {
  static constexpr bool fast = false;
  static constexpr bool records = false;
  bool odd = false;
  __device__ __forceinline__ void check_finite(double) {}
  __device__ __forceinline__ double exp(double x) { return pmp_exp(x); }
  __device__ __forceinline__ double log(double x) { return pmp_log(x); }
  __device__ __forceinline__ double pow(double x, double y) { return pmp_pow(x, y); }  // y > 0
  __device__ __forceinline__ double cbrt(double x) { return pmp_cbrt(x); }
  // log1p(x) and (1 + x)^0.7 sharing one log(1 + x); bit-identical to
  // pmp_log1p(x) and pmp_pow(1. + x, 0.7) for x > -1
  __device__ __forceinline__ void log1p_pow07(double x, double& l1p, double& p07)
  {
    const double u = 1. + x;
    const double lu = pmp_log(u);
    l1p = (fabs(x) < 0.0078125) ? pmp_log1p_core(x) : pmp_log1p_from(x, u, lu);
    p07 = pmp_exp(0.7 * lu);
  }
  __device__ __forceinline__ double div(double a, double b) { return a / b; }
  __device__ __forceinline__ double inv(double b) { return 1. / b; }
  __device__ __forceinline__ Divisor divisor(double b) { return {b, 0.}; }
  __device__ __forceinline__ Divisor divisor_near1(double b) { return {b, 0.}; }
  __device__ __forceinline__ double div(double a, const Divisor& d) { return a / d.b; }
  __device__ __forceinline__ double divk(double a, double b, double) { return a / b; }
};

struct MathFast {
  static constexpr bool fast = true;
  static constexpr bool records = true;  // gathers the box's FP64 gas records
  bool odd = false;

  static constexpr unsigned kRange = 300;
  // v not within 2^+-kRange: zero, subnormal, huge, infinite, NaN, and
  // negative (no divisor of the droplet physics is, but for rare states)
  __device__ __forceinline__ void check_divisor(double v)
  {
    odd |= (unsigned)__double2hiint(v) - ((1023u - kRange) << 20) > (2u * kRange) << 20;
  }
  // v infinite, NaN or above 2^kRange
  __device__ __forceinline__ void check_finite(double v)
  {
    odd |= (__double2hiint(v) & 0x7fffffffu) > (1023u + kRange) << 20;
  }

  __device__ __forceinline__ double exp(double x)
  {
    odd |= (__double2hiint(x) & 0x7fffffff) >= 0x40700000;  // |x| >= 256 or NaN
    constexpr double kMagic = 6755399441055744.0;           // 1.5 2^52
    const double t = __dadd_rn(__dmul_rn(x, PMP_INV_LN2_128), kMagic);
    const int ki = __double2loint(t);
    const double k = __dsub_rn(t, kMagic);
    double r = fma(-k, PMP_LN2_128_HI, x);
    r = fma(-k, PMP_LN2_128_LO, r);
    double p = 8.333333333333333e-03;
    p = fma(p, r, 4.1666666666666664e-02);
    p = fma(p, r, 1.6666666666666666e-01);
    p = fma(p, r, 0.5);
    p = fma(p, r, 1.0);
    p = __dmul_rn(p, r);
    const double e = math_tables().exp2[ki & (PMP_EXP_N - 1)];
    const double v = fma(e, p, e);
    return __hiloint2double(__double2hiint(v) + ((ki >> 7) << 20), __double2loint(v));
  }

  __device__ __forceinline__ double log(double x)
  {
    const int hi = __double2hiint(x);
    const int lo = __double2loint(x);
    odd |= (unsigned)(hi - 0x00100000) >= 0x7fe00000u;  // not positive, normal and finite
    const int mh = (hi & 0x000fffff) | 0x3ff00000;
    const bool upper = ((long long)mh << 32 | (unsigned)lo) > 0x3ff6a09e667f3bcdLL;  // m > sqrt(2)
    const int e = (hi >> 20) - 1023 + (upper ? 1 : 0);
    const double m = __hiloint2double(mh - (upper ? 0x00100000 : 0), lo);
    const double f = __dsub_rn(m, 1.0);  // negative exactly when m was halved
    const int jt = __double2loint(__fma_rz(fabs(f), 128.0, 6755399441055744.0));
    const int j = (upper ? -jt : jt) - PMP_LOG_JMIN;
    const MathTables& t = math_tables();
    const double2 a = t.loga[j];
    const double r = fma(m, a.x, -1.0);
    const double p = pmp_log1p_core(r);
    const double de = __dsub_rn(__hiloint2double(0x43300000, e ^ 0x80000000), 4503601774854144.0);  // e, exactly
    const double h = fma(de, PMP_LN2_HI, a.y);
    const double l = __dadd_rn(fma(de, PMP_LN2_LO, t.logl[j]), p);
    return __dadd_rn(h, l);
  }

  // 1/u to single precision, correctly rounded as pmp_rcp24's division: u's
  // exponent in the middle of the single-precision range, its significand in
  // single precision not all ones (one Newton step from a faithful estimate)
  __device__ __forceinline__ double rcp24(double u)
  {
    const unsigned e2 = (unsigned)(__double2hiint(u) << 1);
    odd |= e2 - ((1023u - 120u) << 21) > 240u << 21;
    const float f = __double2float_rn(u);
    odd |= (__float_as_int(f) & 0x007fffff) == 0x007fffff;
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(f));
    y = __fmaf_rn(y, __fmaf_rn(-f, y, 1.f), y);
    return (double)y;
  }

  __device__ __forceinline__ double pow(double x, double y)
  {
    const bool was = odd;
    const double v = exp(__dmul_rn(y, log(x)));
    odd = x == 0.0 ? was : odd;
    return x == 0.0 ? 0.0 : v;
  }

  __device__ __forceinline__ double cbrt(double x)
  {
    const bool was = odd;
    const double a = fabs(x);
    double y = exp(__dmul_rn(log(a), 1.0 / 3.0));
    const double y2 = __dmul_rn(y, y);
    const double e2 = fma(y, y, -y2);
    double r = fma(y2, y, -a);
    r = fma(e2, y, r);
    y = fma(-r, rcp24(__dmul_rn(3.0, y2)), y);
    odd = x == 0.0 ? was : odd;
    return x == 0.0 ? x : (x < 0.0 ? -y : y);
  }

  __device__ __forceinline__ void log1p_pow07(double x, double& l1p, double& p07)
  {
    const double u = __dadd_rn(1., x);
    const double lu = log(u);
    if (fabs(x) < 0.0078125) {
      l1p = pmp_log1p_core(x);
    } else {
      l1p = fma(__dsub_rn(x, __dsub_rn(u, 1.0)), rcp24(u), lu);  // lu itself where the correction is zero
    }
    p07 = exp(__dmul_rn(0.7, lu));
  }

  // 1/b, b's significand not all ones: the last of three Newton steps is
  // correctly rounded
  __device__ __forceinline__ double rcp(double b)
  {
    check_divisor(b);
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));  // relative error 2^-23
    y = fma(y, fma(-b, y, 1.), y);
    y = fma(y, fma(-b, y, 1.), y);
    return fma(y, fma(-b, y, 1.), y);
  }
  __device__ __forceinline__ bool ones(double b)
  {
    return ((__double2hiint(b) | 0xfff00000u) & (unsigned)__double2loint(b)) == 0xffffffffu;
  }
  __device__ __forceinline__ double inv(double b)
  {
    odd |= ones(b);
    return rcp(b);
  }
  // inv for sums of fractions, which often are 1 - 2^-53: b = 2^k (1 - 2^-53)
  // has 1/b rounded = 2^-k (1 + 2^-52)
  __device__ __forceinline__ double inv_near1(double b)
  {
    const double y = rcp(b);
    return ones(b) ? __hiloint2double(0x7fd00000 - (__double2hiint(b) & 0x7ff00000), 1) : y;
  }
  __device__ __forceinline__ double quotient(double a, double b, double y)
  {
    const double q = __dmul_rn(a, y);
    return fma(fma(-b, q, a), y, q);
  }
  __device__ __forceinline__ Divisor divisor(double b) { return {b, inv(b)}; }
  __device__ __forceinline__ Divisor divisor_near1(double b) { return {b, inv_near1(b)}; }
  __device__ __forceinline__ double div(double a, const Divisor& d) { return quotient(a, d.b, d.y); }
  __device__ __forceinline__ double div(double a, double b) { return quotient(a, b, inv(b)); }
  // y: the host's 1. / b, b in the middle of the range
  __device__ __forceinline__ double divk(double a, double b, double y) { return quotient(a, b, y); }
};

// the same where the update gathers the caller's planes (no FP64 records)
struct MathFastPlanes : MathFast {
  static constexpr bool records = false;
};

}  // namespace pmp
