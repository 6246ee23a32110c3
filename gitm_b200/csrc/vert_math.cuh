// vert_math.cuh -- the FP64 reciprocal of the friction solves, as plain
// multiply-adds.
//
// CUDA's division ends in a range test with a slow path behind a branch; the
// six pivots of a friction solve are a serial chain, and each branch ends the
// block the compiler can schedule over.  rcp_nr refines PTX's documented
// rcp.approx.ftz.f64 (relative error 2^-23) with two Newton-Raphson steps:
// four FP64 instructions.  The header also compiles as plain C++, for
// tests/test_math.py.
#pragma once

#include <cstdint>
#ifdef __CUDACC__
#define GV_MATH __device__ __forceinline__
#else
#include <cmath>
#include <cstring>
#define GV_MATH inline
#endif

namespace gv {

#ifdef __CUDACC__
GV_MATH double m_fma(double a, double b, double c) { return fma(a, b, c); }
GV_MATH double rcp_seed(double a) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(a));
  return r;
}
#else
GV_MATH double m_fma(double a, double b, double c) { return std::fma(a, b, c); }
// a seed of the documented accuracy where there is no GPU: 22 bits of 1 / a
GV_MATH double rcp_seed(double a) {
  double r = 1.0 / a;
  uint64_t u;
  std::memcpy(&u, &r, 8);
  u &= 0xffffffffc0000000ull;
  std::memcpy(&r, &u, 8);
  return r;
}
#endif

// 1 / a.  Relative error at most 1 ulp for |a| in [2^-1020, 2^1020]; a zero,
// subnormal, infinite or NaN argument gives a result that is not finite.
GV_MATH double rcp_nr(double a) {
  double r = rcp_seed(a);
  r = m_fma(r, m_fma(-a, r, 1.0), r);
  return m_fma(r, m_fma(-a, r, 1.0), r);
}

}  // namespace gv
