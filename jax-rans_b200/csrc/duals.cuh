// A value with N tangents: N columns of a Jacobian from one evaluation of the pointwise
// physics (physics.cuh, device3d.cuh).  The value's arithmetic is the plain path's,
// operation for operation, so every branch is the one the residual takes; the JVP rules
// are Dual's.  A quotient's tangents share one reciprocal of the divisor and a root's one
// reciprocal of the root: FP64 divisions and roots are most of a flux's issue slots, and
// with one tangent at a time (Dual) each column pays for them again.
#pragma once
#include "physics.cuh"

namespace jr {

template <int N> struct Duals {
  double v, d[N];
};

#define JR_HD __host__ __device__ __forceinline__

template <int N> JR_HD double val(const Duals<N>& x) { return x.v; }
template <int N> JR_HD Duals<N> duals_cst(double x) {
  Duals<N> r;
  r.v = x;
#pragma unroll
  for (int k = 0; k < N; ++k) r.d[k] = 0.0;
  return r;
}
template <> JR_HD Duals<2> cst<Duals<2>>(double x) { return duals_cst<2>(x); }
template <> JR_HD Duals<3> cst<Duals<3>>(double x) { return duals_cst<3>(x); }
template <> JR_HD Duals<4> cst<Duals<4>>(double x) { return duals_cst<4>(x); }

// r.v = VALUE, r.d[k] = TANGENT for every k
#define JR_DUALS(VALUE, TANGENT)          \
  Duals<N> r;                             \
  r.v = VALUE;                            \
  _Pragma("unroll") for (int k = 0; k < N; ++k) r.d[k] = TANGENT; \
  return r

template <int N> JR_HD Duals<N> operator+(const Duals<N>& a, const Duals<N>& b) { JR_DUALS(a.v + b.v, a.d[k] + b.d[k]); }
template <int N> JR_HD Duals<N> operator-(const Duals<N>& a, const Duals<N>& b) { JR_DUALS(a.v - b.v, a.d[k] - b.d[k]); }
template <int N> JR_HD Duals<N> operator-(const Duals<N>& a) { JR_DUALS(-a.v, -a.d[k]); }
template <int N> JR_HD Duals<N> operator*(const Duals<N>& a, const Duals<N>& b) {
  JR_DUALS(a.v * b.v, a.d[k] * b.v + a.v * b.d[k]);
}
template <int N> JR_HD Duals<N> operator/(const Duals<N>& a, const Duals<N>& b) {
  const double q = a.v / b.v, inv = 1.0 / b.v;
  JR_DUALS(q, (a.d[k] - q * b.d[k]) * inv);
}
template <int N> JR_HD Duals<N> operator+(const Duals<N>& a, double b) { JR_DUALS(a.v + b, a.d[k]); }
template <int N> JR_HD Duals<N> operator+(double a, const Duals<N>& b) { JR_DUALS(a + b.v, b.d[k]); }
template <int N> JR_HD Duals<N> operator-(const Duals<N>& a, double b) { JR_DUALS(a.v - b, a.d[k]); }
template <int N> JR_HD Duals<N> operator-(double a, const Duals<N>& b) { JR_DUALS(a - b.v, -b.d[k]); }
template <int N> JR_HD Duals<N> operator*(const Duals<N>& a, double b) { JR_DUALS(a.v * b, a.d[k] * b); }
template <int N> JR_HD Duals<N> operator*(double a, const Duals<N>& b) { JR_DUALS(a * b.v, a * b.d[k]); }
template <int N> JR_HD Duals<N> operator/(const Duals<N>& a, double b) {
  const double inv = 1.0 / b;
  JR_DUALS(a.v / b, a.d[k] * inv);
}
template <int N> JR_HD Duals<N> operator/(double a, const Duals<N>& b) {
  const double q = a / b.v, f = -q / b.v;
  JR_DUALS(q, f * b.d[k]);
}
template <int N> JR_HD Duals<N> dsqrt(const Duals<N>& x) {
  const double s = sqrt(x.v), f = 0.5 / s;
  JR_DUALS(s, x.d[k] * f);
}
template <int N> JR_HD Duals<N> dpow(const Duals<N>& x, double c) {
  const double f = c * pow(x.v, c - 1.0);
  JR_DUALS(pow(x.v, c), x.d[k] * f);
}
template <int N> JR_HD Duals<N> dabs(const Duals<N>& x) { return x.v >= 0.0 ? x : -x; }
template <int N> JR_HD Duals<N> dmax(const Duals<N>& a, const Duals<N>& b) {
  const bool more = a.v > b.v, less = b.v > a.v;
  JR_DUALS(more ? a.v : (less ? b.v : a.v), more ? a.d[k] : (less ? b.d[k] : 0.5 * (a.d[k] + b.d[k])));
}
template <int N> JR_HD Duals<N> dmin(const Duals<N>& a, const Duals<N>& b) {
  const bool less = a.v < b.v, more = b.v < a.v;
  JR_DUALS(less ? a.v : (more ? b.v : a.v), less ? a.d[k] : (more ? b.d[k] : 0.5 * (a.d[k] + b.d[k])));
}
template <int N> JR_HD Duals<N> dmax(const Duals<N>& a, double b) { return dmax(a, duals_cst<N>(b)); }
template <int N> JR_HD Duals<N> dmin(const Duals<N>& a, double b) { return dmin(a, duals_cst<N>(b)); }
template <int N> JR_HD Duals<N> sel(bool c, const Duals<N>& a, double b) { return c ? a : duals_cst<N>(b); }
template <int N> JR_HD Duals<N> sel(bool c, double a, const Duals<N>& b) { return c ? duals_cst<N>(a) : b; }

#undef JR_DUALS
#undef JR_HD

}  // namespace jr
