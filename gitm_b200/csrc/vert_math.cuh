// vert_math.cuh -- FP64 exp, log and reciprocal for the stage kernels.
//
// What bounds a stage is the number of instructions its warps issue and the
// latency of their FP64 chains, and the calls of CUDA's exp and log in a loop
// over species run one after the other: seven logarithms take one warp 1,900
// cycles, in a batch 840.  The batches here run N arguments side by side with
// one range test for all: 18 instructions per exp (15 FP64), 32 per log (23),
// 5 per reciprocal.
//
// Written from the mathematics and published methods.  exp's range reduction
// is Cody and Waite's (Software Manual for the Elementary Functions, 1980:
// ln 2 in two parts).  log's reduction to mantissas in [sqrt(1/2), sqrt(2)) by
// an offset of the exponent field, and the arrangement f - s (f - z p) that
// keeps f's bits, are those of FreeBSD's msun (e_log.c, from Sun's fdlibm; musl
// has them from there).  The polynomials are Chebyshev interpolants of (e^r - 1
// - r) / r^2 on |r| <= 0.347 (truncation 1.7e-17 relative) and of the atanh
// series on those mantissas (4.7e-18), computed for this file; the reciprocal
// refines PTX's documented rcp.approx.ftz.f64 with Newton-Raphson steps.  Error
// against the exact value, on the device and as plain C++: below 1 ulp (exp,
// log, reciprocal); tests/test_gpu_math.py and tests/test_math.py.
#pragma once

#include <cstdint>
#ifdef __CUDACC__
#define GV_MATH __device__ __forceinline__
#define GV_UNROLL _Pragma("unroll")
#else
#include <cmath>
#include <cstring>
using std::fabs;
#define GV_MATH inline
#define GV_UNROLL
#endif

namespace gv {

#ifdef __CUDACC__
GV_MATH int m_hi(double x) { return __double2hiint(x); }
GV_MATH int m_lo(double x) { return __double2loint(x); }
GV_MATH double m_make(int hi, int lo) { return __hiloint2double(hi, lo); }
GV_MATH double m_fma(double a, double b, double c) { return fma(a, b, c); }
GV_MATH double rcp_seed(double a) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(a));
  return r;
}
#else
GV_MATH int m_hi(double x) {
  uint64_t u;
  std::memcpy(&u, &x, 8);
  return int(uint32_t(u >> 32));
}
GV_MATH int m_lo(double x) {
  uint64_t u;
  std::memcpy(&u, &x, 8);
  return int(uint32_t(u));
}
GV_MATH double m_make(int hi, int lo) {
  const uint64_t u = (uint64_t(uint32_t(hi)) << 32) | uint32_t(lo);
  double x;
  std::memcpy(&x, &u, 8);
  return x;
}
GV_MATH double m_fma(double a, double b, double c) { return std::fma(a, b, c); }
// a seed of the documented accuracy (20 bits) where there is no GPU
GV_MATH double rcp_seed(double a) {
  const double r = 1.0 / a;
  return m_make(m_hi(r), 0);
}
#endif

// The constants are read from constant memory, where an FP64 instruction
// takes them as an operand.
#ifdef __CUDACC__
static __constant__ double
#else
static const double
#endif
    m_k[] = {
        1.4426950408889634,      // 0: log2 e
        0.6931471805582987,      // 1: ln 2 to 38 fraction bits: n times it is exact
        1.6465949582897082e-12,  // 2: the rest of ln 2
        6755399441055744.0,      // 3: 1.5 * 2^52: adding it rounds to an integer
        // 4..13: (e^r - 1 - r) / r^2, highest power first
        2.5100494788905042e-08, 2.76202305675069e-07, 2.7557268229963227e-06, 2.4801520996825697e-05,
        0.00019841269863201828, 0.0013888888917406447, 0.008333333333330032, 0.04166666666662374,
        0.16666666666666669, 0.5000000000000001,
        // 14..20: (2 atanh(s) - 2 s) / s^3 in s^2, highest power first
        0.1461916477718642, 0.1533150172120742, 0.18182895746801428, 0.22222211043822487,
        0.28571428626533335, 0.3999999999989827, 0.666666666666667};

// 1 / a.  Relative error below 1 ulp for |a| in [2^-1020, 2^1020]; outside
// (0, infinities, NaN, subnormals) the result is not finite or NaN.
GV_MATH double rcp_nr(double a) {
  double r = rcp_seed(a);
  r = m_fma(r, m_fma(-a, r, 1.0), r);
  return m_fma(r, m_fma(-a, r, 1.0), r);
}

// ModLimiter.f90:16-36: on same-sign slopes the smallest magnitude of beta u,
// beta d and (u + d) / 2 carries the common sign (the reference's min of the
// three when both are positive and max when both are negative, the same values
// since negation is exact and rounding monotonic: min(beta |u|, beta |d|) =
// beta min(|u|, |d|)); 0 otherwise.  Selects on plain comparisons: fmin and the
// four comparisons with zero took about twice the instructions.  A NaN goes the
// way of the reference's comparisons, which pass it over or give zero, so it
// does not spread along the column (a branch for it cost 5 % of a step; this
// form costs nothing that shows).
GV_MATH double limiter_mc(double u, double d, double beta) {
  const double au = fabs(u), ad = fabs(d);
  const double t = beta * (au < ad ? au : ad);
  const double s = (u + d) * 0.5, as = fabs(s);
  const double m = as < t ? as : t;
  const int neg = u > 0.0 ? 0 : int(0x80000000u);
  const bool on = m_make(m_hi(d) ^ neg, m_lo(d)) > 0.0;  // d has the slopes' sign
  return on ? m_make(m_hi(m) | neg, m_lo(m)) : 0.0;
}

// CUDA's own functions, out of line: the batches below take them for the
// arguments outside their fast range.
#ifdef __CUDACC__
static __device__ __noinline__ double exp_any(double x) { return exp(x); }
static __device__ __noinline__ double log_any(double x) { return log(x); }
#else
inline double exp_any(double x) { return std::exp(x); }
inline double log_any(double x) { return std::log(x); }
#endif

// Whether the far branch is taken.  WARP: by whole warps (the caller's warp
// is converged and has to stay so), else lane by lane.
template <bool WARP>
GV_MATH bool m_any(bool far) {
#ifdef __CUDACC__
  if (WARP) return __any_sync(0xffffffffu, far);
#endif
  return far;
}

// The batches run step by step over their N arguments: in source order N
// independent chains side by side, which is also how they are issued (a loop
// over whole calls came out one call after the other).

// y = e^x for every x.
template <int N, bool WARP = false>
GV_MATH void exp_n(const double (&x)[N], double (&y)[N]) {
  double r[N], p[N];
  int n[N], top = 0;
  GV_UNROLL for (int j = 0; j < N; ++j) {
    const int ax = m_hi(x[j]) & 0x7fffffff;
    top = ax > top ? ax : top;
    p[j] = m_fma(x[j], m_k[0], m_k[3]);
  }
  GV_UNROLL for (int j = 0; j < N; ++j) {
    n[j] = m_lo(p[j]);
    p[j] = p[j] - m_k[3];
  }
  GV_UNROLL for (int j = 0; j < N; ++j) r[j] = m_fma(-p[j], m_k[1], x[j]);
  GV_UNROLL for (int j = 0; j < N; ++j) r[j] = m_fma(-p[j], m_k[2], r[j]);
  GV_UNROLL for (int j = 0; j < N; ++j) p[j] = m_fma(m_k[4], r[j], m_k[5]);
  GV_UNROLL for (int k = 6; k < 14; ++k)
    GV_UNROLL for (int j = 0; j < N; ++j) p[j] = m_fma(p[j], r[j], m_k[k]);
  GV_UNROLL for (int j = 0; j < N; ++j) p[j] = m_fma(p[j], r[j], 1.0);
  GV_UNROLL for (int j = 0; j < N; ++j) p[j] = m_fma(p[j], r[j], 1.0);
  // times 2^n in the exponent field: a normal number for |x| < 708
  GV_UNROLL for (int j = 0; j < N; ++j) y[j] = m_make(m_hi(p[j]) + (n[j] << 20), m_lo(p[j]));
  const bool far = top >= 0x40862000;  // |x| >= 708, infinities, NaN
  if (m_any<WARP>(far)) {
    GV_UNROLL for (int j = 0; j < N; ++j) {
      const double v = exp_any(x[j]);
      y[j] = far ? v : y[j];
    }
  }
}

// y = log x for every x.
template <int N, bool WARP = false>
GV_MATH void log_n(const double (&x)[N], double (&y)[N]) {
  double f[N], d[N], r[N], s[N], z[N], p[N];
  int e[N];
  bool far = false;  // not a normal positive number
  GV_UNROLL for (int j = 0; j < N; ++j) {
    // mantissa in [sqrt(1/2), sqrt(2)): offset the exponent field by that of sqrt(1/2)
    far = far || unsigned(m_hi(x[j])) - 0x00100000u >= 0x7fe00000u;
    const int hm = m_hi(x[j]) + (0x3ff00000 - 0x3fe6a09e);
    e[j] = (hm >> 20) - 1023;
    const double m = m_make((hm & 0x000fffff) + 0x3fe6a09e, m_lo(x[j]));
    f[j] = m - 1.0;
    d[j] = m + 1.0;
  }
  // s = f / d, the quotient corrected by its residual
  GV_UNROLL for (int j = 0; j < N; ++j) r[j] = rcp_seed(d[j]);
  GV_UNROLL for (int j = 0; j < N; ++j) s[j] = m_fma(-d[j], r[j], 1.0);
  GV_UNROLL for (int j = 0; j < N; ++j) r[j] = m_fma(r[j], s[j], r[j]);
  GV_UNROLL for (int j = 0; j < N; ++j) s[j] = f[j] * r[j];
  GV_UNROLL for (int j = 0; j < N; ++j) z[j] = m_fma(-d[j], s[j], f[j]);
  GV_UNROLL for (int j = 0; j < N; ++j) s[j] = m_fma(z[j], r[j], s[j]);
  GV_UNROLL for (int j = 0; j < N; ++j) z[j] = s[j] * s[j];
  GV_UNROLL for (int j = 0; j < N; ++j) p[j] = m_fma(m_k[14], z[j], m_k[15]);
  GV_UNROLL for (int k = 16; k < 21; ++k)
    GV_UNROLL for (int j = 0; j < N; ++j) p[j] = m_fma(p[j], z[j], m_k[k]);
  // log m = 2 s + s z p, with f = 2 s + s f: f - s (f - z p) keeps f's bits
  GV_UNROLL for (int j = 0; j < N; ++j) p[j] = m_fma(-z[j], p[j], f[j]);
  GV_UNROLL for (int j = 0; j < N; ++j) p[j] = -s[j] * p[j];
  GV_UNROLL for (int j = 0; j < N; ++j) {
    const double ed = m_make(0x43300000, e[j] ^ int(0x80000000u)) - 4503601774854144.0;  // e as a double
    // e ln2 + f with its rounding error carried (|e ln2| > |f| or e = 0)
    const double eh = ed * m_k[1];
    const double b = eh + f[j];
    y[j] = b + ((f[j] - (b - eh)) + m_fma(ed, m_k[2], p[j]));
  }
  if (m_any<WARP>(far)) {
    GV_UNROLL for (int j = 0; j < N; ++j) {
      const double v = log_any(x[j]);
      y[j] = far ? v : y[j];
    }
  }
}

GV_MATH double exp_sl(double x) {
  const double a[1] = {x};
  double y[1];
  exp_n(a, y);
  return y[0];
}

GV_MATH double log_sl(double x) {
  const double a[1] = {x};
  double y[1];
  log_n(a, y);
  return y[0];
}

}  // namespace gv
