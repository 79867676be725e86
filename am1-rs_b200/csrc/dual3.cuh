// Forward-mode dual numbers.  D3: a value and its gradient with respect to the pair displacement (delta_x,
// delta_y, delta_z).  D1: a value and its derivative with respect to the distance r, for the quantities that
// depend on r alone (the local-frame integrals and overlaps, the core-core energy), whose gradient is that derivative
// times the unit vector of the displacement (lift): a third of the derivative arithmetic.  The integral and
// overlap templates of integrals_t.cuh instantiated with them give the exact derivatives of the quantities the
// SCF evaluates (the reference's Dual, src/dual.rs, carries three components throughout for the same
// purpose).  Only the operations the integral code uses are defined.
#pragma once

#include <cuda_runtime.h>

namespace am1 {

template <int K>
struct Dual {
    double v;
    double d[K];
};
using D1 = Dual<1>;
using D3 = Dual<3>;

__device__ __forceinline__ double val(double x) { return x; }
template <int K>
__device__ __forceinline__ double val(const Dual<K>& x) { return x.v; }

// v, with derivative components f(k)
template <int K, class F>
__device__ __forceinline__ Dual<K> dual_of(double v, F&& f) {
    Dual<K> r;
    r.v = v;
#pragma unroll
    for (int k = 0; k < K; ++k) r.d[k] = f(k);
    return r;
}

#define AM1_DUAL_OP template <int K> __device__ __forceinline__ Dual<K>
AM1_DUAL_OP operator+(const Dual<K>& a, const Dual<K>& b) { return dual_of<K>(a.v + b.v, [&](int k) { return a.d[k] + b.d[k]; }); }
AM1_DUAL_OP operator-(const Dual<K>& a, const Dual<K>& b) { return dual_of<K>(a.v - b.v, [&](int k) { return a.d[k] - b.d[k]; }); }
AM1_DUAL_OP operator-(const Dual<K>& a) { return dual_of<K>(-a.v, [&](int k) { return -a.d[k]; }); }
AM1_DUAL_OP operator*(const Dual<K>& a, const Dual<K>& b) {
    return dual_of<K>(a.v * b.v, [&](int k) { return a.d[k] * b.v + a.v * b.d[k]; });
}
AM1_DUAL_OP operator/(const Dual<K>& a, const Dual<K>& b) {
    const double q = a.v / b.v, ib = 1.0 / b.v;
    return dual_of<K>(q, [&](int k) { return (a.d[k] - q * b.d[k]) * ib; });
}
AM1_DUAL_OP operator+(const Dual<K>& a, double b) { return dual_of<K>(a.v + b, [&](int k) { return a.d[k]; }); }
AM1_DUAL_OP operator+(double a, const Dual<K>& b) { return b + a; }
AM1_DUAL_OP operator-(const Dual<K>& a, double b) { return dual_of<K>(a.v - b, [&](int k) { return a.d[k]; }); }
AM1_DUAL_OP operator-(double a, const Dual<K>& b) { return dual_of<K>(a - b.v, [&](int k) { return -b.d[k]; }); }
AM1_DUAL_OP operator*(const Dual<K>& a, double b) { return dual_of<K>(a.v * b, [&](int k) { return a.d[k] * b; }); }
AM1_DUAL_OP operator*(double a, const Dual<K>& b) { return b * a; }
AM1_DUAL_OP operator/(const Dual<K>& a, double b) { return dual_of<K>(a.v / b, [&](int k) { return a.d[k] / b; }); }
AM1_DUAL_OP operator/(double a, const Dual<K>& b) {
    const double q = a / b.v, s = -q / b.v;
    return dual_of<K>(q, [&](int k) { return s * b.d[k]; });
}
template <int K>
__device__ __forceinline__ Dual<K>& operator+=(Dual<K>& a, const Dual<K>& b) { return a = a + b; }
template <int K>
__device__ __forceinline__ Dual<K>& operator*=(Dual<K>& a, const Dual<K>& b) { return a = a * b; }

// The double overloads forward to the CUDA math functions: inside this namespace the dual overloads
// below would otherwise hide them.
__device__ __forceinline__ double exp(double x) { return ::exp(x); }
__device__ __forceinline__ double sqrt(double x) { return ::sqrt(x); }
__device__ __forceinline__ double pow(double x, double p) { return ::pow(x, p); }

// f(x) with f' = df at x: the chain rule on the components
AM1_DUAL_OP dual_chain(const Dual<K>& x, double f, double df) { return dual_of<K>(f, [&](int k) { return df * x.d[k]; }); }

AM1_DUAL_OP exp(const Dual<K>& x) {
    const double e = ::exp(x.v);
    return dual_chain(x, e, e);
}
AM1_DUAL_OP sqrt(const Dual<K>& x) {
    const double s = ::sqrt(x.v);
    return dual_chain(x, s, 0.5 / s);
}
// x^p for a constant p (x > 0)
AM1_DUAL_OP pow(const Dual<K>& x, double p) {
    const double f = ::pow(x.v, p);
    return dual_chain(x, f, p * f / x.v);
}
#undef AM1_DUAL_OP

// A quantity of r in the arithmetic of the displacement: u, the unit vector of the displacement (unused for
// plain values).
__device__ __forceinline__ double lift(double x, const double*) { return x; }
__device__ __forceinline__ D3 lift(const D1& x, const double u[3]) { return D3{x.v, {x.d[0] * u[0], x.d[0] * u[1], x.d[0] * u[2]}}; }

}  // namespace am1
