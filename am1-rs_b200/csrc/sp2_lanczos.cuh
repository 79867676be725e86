// The small tridiagonal problems behind the Lanczos spectral bounds, shared by the bounds kernels
// (k_sp2.cu) and the one-launch purification (k_sp2_fused.cu).
#pragma once

#include <cuda_runtime.h>

namespace am1 {

constexpr int SP2_LANCZOS = 12;
// largest widening of a reused spectral interval, as a fraction of the width of the last Lanczos run's
constexpr double SP2_REUSE_FRAC = 0.01;
constexpr int SP2_BOUND_THREADS = 512;

// Eigenvalues of T (m x m, diagonal a, off-diagonal b) below x.
__device__ inline int lz_count(const double* a, const double* b, int m, double x) {
    int c = 0;
    double q = a[0] - x;
    if (q < 0.0) ++c;
    for (int i = 1; i < m; ++i) {
        q = a[i] - x - b[i - 1] * b[i - 1] / (q == 0.0 ? 1e-300 : q);
        if (q < 0.0) ++c;
    }
    return c;
}

// k-th smallest eigenvalue of T by bisection inside [lo, hi].
__device__ inline double lz_eig(const double* a, const double* b, int m, int k, double lo, double hi) {
    for (int it = 0; it < 200; ++it) {
        const double mid = 0.5 * (lo + hi);
        if (!(mid > lo && mid < hi)) break;
        if (lz_count(a, b, m, mid) <= k) lo = mid;
        else hi = mid;
    }
    return 0.5 * (lo + hi);
}

// The same eigenvalue by one warp: 32-way multisection, each round 31 Sturm counts at interior
// points of [lo, hi] on the lanes and the interval narrowed to the gap where the count passes k (a
// factor 32 per round; 11 rounds reach the rounding level of the bisection).  Every lane of the warp
// calls it and gets the same value.
__device__ inline double lz_eig_warp(const double* a, const double* b, int m, int k, double lo, double hi) {
    const int lane = threadIdx.x & 31;
    for (int round = 0; round < 11; ++round) {
        const double h = (hi - lo) * (1.0 / 32.0);
        if (!(h > 0.0)) break;
        const double x = lo + h * (lane + 1);
        const bool below = lane < 31 && lz_count(a, b, m, x) <= k;  // x <= the k-th eigenvalue
        const unsigned ball = __ballot_sync(0xffffffffu, below);
        const int j = ball ? 31 - __clz(ball) : -1;  // the last interior point still below it
        const double nlo = j >= 0 ? lo + h * (j + 1) : lo;
        const double nhi = j + 2 <= 31 ? lo + h * (j + 2) : hi;
        lo = nlo;
        hi = nhi;
    }
    return 0.5 * (lo + hi);
}

// |last component| of the unit eigenvector of T for an exterior eigenvalue: inverse iteration
// with the shift sigma just outside the spectrum, so T - sigma I is definite and the
// tridiagonal solve needs no pivoting.  The elimination is the same in each of the three iterations and
// is done once; the loops are unrolled to SP2_LANCZOS so that every vector stays in registers (in local
// memory, with the elimination repeated, the two ends' calls took 12 of the 23 us behind a Lanczos run).
__device__ inline double lz_last_component(const double* a, const double* b, int m, double sigma) {
    double x[SP2_LANCZOS], cp[SP2_LANCZOS], rp[SP2_LANCZOS], den[SP2_LANCZOS], be[SP2_LANCZOS];
    den[0] = a[0] - sigma;
    be[0] = m > 1 ? b[0] : 0.0;
    cp[0] = m > 1 ? be[0] / den[0] : 0.0;
#pragma unroll
    for (int i = 1; i < SP2_LANCZOS; ++i) {
        den[i] = 1.0;
        be[i] = cp[i] = 0.0;
        if (i < m) {
            be[i] = i + 1 < m ? b[i] : 0.0;
            den[i] = a[i] - sigma - be[i - 1] * cp[i - 1];
            cp[i] = i + 1 < m ? be[i] / den[i] : 0.0;
        }
    }
#pragma unroll
    for (int i = 0; i < SP2_LANCZOS; ++i) x[i] = 1.0;
    double last = 1.0;
#pragma unroll 1
    for (int it = 0; it < 3; ++it) {
        rp[0] = x[0] / den[0];
#pragma unroll
        for (int i = 1; i < SP2_LANCZOS; ++i) {
            rp[i] = 0.0;
            if (i < m) rp[i] = (x[i] - be[i - 1] * rp[i - 1]) / den[i];
        }
        double nrm = 0.0;
#pragma unroll
        for (int i = SP2_LANCZOS - 1; i >= 0; --i)
            if (i < m) x[i] = i == m - 1 ? rp[i] : rp[i] - cp[i] * x[i + 1 < SP2_LANCZOS ? i + 1 : i];
#pragma unroll
        for (int i = 0; i < SP2_LANCZOS; ++i)
            if (i < m) nrm += x[i] * x[i];
        nrm = sqrt(nrm);
        if (!(nrm > 0.0) || !isfinite(nrm)) return 1.0;
#pragma unroll
        for (int i = 0; i < SP2_LANCZOS; ++i)
            if (i < m) {
                x[i] /= nrm;
                if (i == m - 1) last = x[i];
            }
    }
    return fabs(last);
}

}  // namespace am1
