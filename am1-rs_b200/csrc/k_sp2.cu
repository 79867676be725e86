// Density matrix of the SCF step by trace-correcting purification (SP2), batched.
//
// The SCF needs only P = w * (projector onto the n_occ lowest eigenvectors of F*), which is what
// am1-rs builds from the eigenvectors (src/scf.rs:654-661: symmetric_eigen then
// density_from_coeff).  SP2 (Niklasson, Phys. Rev. B 66, 155115 (2002)) reaches the same
// projector with matrix products only:
//     X0 = (e_max I - F*) / (e_max - e_min)         (Gershgorin bounds, spectrum mapped into [0,1])
//     X <- X^2  or  X <- 2X - X^2                   (whichever brings tr X closer to n_occ)
// until X is idempotent to rounding.  Each step is one symmetric FP64 product X.X on the tensor
// cores (mma.sync m16n8k8 f64), upper-triangle tiles only, mirrored in the epilogue, which also
// folds in the choice of branch and the tile's share of tr X and ||X||_F^2 (= tr X^2 for the
// next step's decision).  No eigenvectors, no fine-grained synchronisation: every step is one
// launch over all (molecule, channel) tiles of the batch.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "am1gpu_internal.h"
#include "dmma_gemm.cuh"
#include "kernels.h"
#include "sp2_lanczos.cuh"

namespace am1 {

namespace cg = cooperative_groups;


// Spectral bounds [e_min, e_max] of F* for the SP2 mapping.  The number of purification steps
// grows with the width of the interval, and the Gershgorin interval of an NDDO Fock matrix is
// about twice the true spectral width (the row sums over the many small long-range elements), so
// the bounds come from a short Lanczos run (SP2_LANCZOS steps from a fixed start vector, no
// reorthogonalisation: only the extreme Ritz values are used):
//     e_max = min(Gershgorin max, theta_max + r_max + 0.005 w)
//     e_min = max(Gershgorin min, theta_min - r_min - 0.005 w)
// with r = |beta_m s_m| the residual of the extreme Ritz pair (s from inverse iteration on the
// Lanczos tridiagonal T) and w = theta_max - theta_min.  An eigenvalue left slightly outside
// the interval maps just outside [0, 1], where the trace-correcting steps pull it back; a run
// that still fails to converge falls back to the eigensolver.  One CTA per channel.
__device__ double bounds_block_sum(double v, double* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double t = 0.0;
    for (int w = 0; w < SP2_BOUND_THREADS / 32; ++w) t += red[w];
    return t;
}

__global__ void __launch_bounds__(SP2_BOUND_THREADS, 2) k_sp2_bounds(const Sp2Job* __restrict__ jobs, const MolState* __restrict__ st) {
    const Sp2Job jb = jobs[blockIdx.x];
    if (!st[jb.mol].active || !jb.fallback || sp2_fused_now(jb, st[jb.mol].lowp)) return;  // large matrices: k_sp2_bounds_big
    const int n = jb.n;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NW = SP2_BOUND_THREADS / 32;
    extern __shared__ double lz[];
    double* q = lz;        // current Lanczos vector
    double* qp = lz + n;   // previous one
    double* w = lz + 2 * n;
    __shared__ double red[NW];
    __shared__ double alpha[SP2_LANCZOS], beta[SP2_LANCZOS];
    // Gershgorin interval (rows of F*)
    __shared__ double gred[2][NW];
    double glo = 1e300, ghi = -1e300;
    for (int i = tid; i < n; i += SP2_BOUND_THREADS) {
        glo = fmin(glo, jb.rowmin[i]);
        ghi = fmax(ghi, jb.rowmax[i]);
    }
    for (int o = 16; o > 0; o >>= 1) {
        glo = fmin(glo, __shfl_xor_sync(0xffffffffu, glo, o));
        ghi = fmax(ghi, __shfl_xor_sync(0xffffffffu, ghi, o));
    }
    if (lane == 0) {
        gred[0][warp] = glo;
        gred[1][warp] = ghi;
    }
    // From the second SCF iteration on, F* has moved by delta = ||F* - F*_previous||_F from the matrix
    // of the previous interval, and no eigenvalue moves further than that (Weyl's inequality,
    // |lambda_i(A + E) - lambda_i(A)| <= ||E||_2 <= ||E||_F).  While the widening added since the last
    // Lanczos run stays below SP2_REUSE_FRAC of that run's width, the previous interval widened by
    // delta on both sides (and capped by the Gershgorin interval of F*) is taken instead of a new run.
    const bool may_reuse = jb.rowdf != nullptr && st[jb.mol].iter > 0;
    const double b_lo = jb.bounds[0], b_hi = jb.bounds[1], b_slack = jb.bounds[2], b_width = jb.bounds[3];
    double dsum = 0.0;
    if (may_reuse)
        for (int i = tid; i < n; i += SP2_BOUND_THREADS) dsum += jb.rowdf[i];
    dsum = bounds_block_sum(dsum, red);  // its barriers also publish gred
    if (may_reuse) {
        double rlo = gred[0][0], rhi = gred[1][0];
        for (int v = 1; v < NW; ++v) {
            rlo = fmin(rlo, gred[0][v]);
            rhi = fmax(rhi, gred[1][v]);
        }
        const double delta = sqrt(dsum) * (1.0 + 1e-12);
        const double slack = b_slack + delta;
        const double lo = fmax(b_lo - delta, rlo), hi = fmin(b_hi + delta, rhi);
        if (isfinite(slack) && b_width > 0.0 && slack <= SP2_REUSE_FRAC * b_width && hi > lo) {
            __syncthreads();  // every thread has read the previous interval
            if (tid == 0) {
                jb.bounds[0] = lo;
                jb.bounds[1] = hi;
                jb.bounds[2] = slack;
            }
            return;
        }
    }
    // fixed start vector, normalised
    double nq = 0.0;
    for (int i = tid; i < n; i += SP2_BOUND_THREADS) {
        const double x = cos(0.7 * i + 0.3) + 0.5;
        q[i] = x;
        qp[i] = 0.0;
        nq += x * x;
    }
    nq = bounds_block_sum(nq, red);  // its barriers also publish gred
    glo = gred[0][0];
    ghi = gred[1][0];
    for (int v = 1; v < NW; ++v) {
        glo = fmin(glo, gred[0][v]);
        ghi = fmax(ghi, gred[1][v]);
    }
    const double inq = 1.0 / sqrt(nq);
    for (int i = tid; i < n; i += SP2_BOUND_THREADS) q[i] *= inq;
    __syncthreads();
    const int K = min(SP2_LANCZOS, n);
    const bool pairs = (n & 1) == 0 && (reinterpret_cast<uintptr_t>(jb.F) & 15) == 0;
    int m = 0;
    double bprev = 0.0;
    for (int j = 0; j < K; ++j) {
        // w = F q: eight lanes per row, so every warp has four rows' loads in flight; rows of even
        // length on 16-byte boundaries are read as pairs (16-byte loads, two partial sums per lane)
        const int sub = lane >> 3, sl = lane & 7;
        for (int r0 = 4 * warp; r0 < n; r0 += 4 * NW) {
            const int r = r0 + sub;
            double acc = 0.0;
            if (r < n) {
                const double* Fr = jb.F + (long long)r * n;
                if (pairs) {
                    const double2* F2 = reinterpret_cast<const double2*>(Fr);
                    const double2* q2 = reinterpret_cast<const double2*>(q);
                    double acc1 = 0.0;
#pragma unroll 4
                    for (int c = sl; c < n / 2; c += 8) {
                        const double2 f = F2[c], x = q2[c];
                        acc = fma(f.x, x.x, acc);
                        acc1 = fma(f.y, x.y, acc1);
                    }
                    acc += acc1;
                } else {
                    for (int c = sl; c < n; c += 8) acc = fma(Fr[c], q[c], acc);
                }
            }
            for (int o = 4; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (sl == 0 && r < n) w[r] = acc;
        }
        __syncthreads();
        double part = 0.0;
        for (int i = tid; i < n; i += SP2_BOUND_THREADS) part += q[i] * w[i];
        const double a = bounds_block_sum(part, red);
        part = 0.0;
        for (int i = tid; i < n; i += SP2_BOUND_THREADS) {
            const double x = w[i] - a * q[i] - bprev * qp[i];
            w[i] = x;
            part += x * x;
        }
        const double bnorm = sqrt(bounds_block_sum(part, red));
        if (tid == 0) {
            alpha[j] = a;
            beta[j] = bnorm;
        }
        m = j + 1;
        if (!(bnorm > 1e-12 * fmax(fabs(a), 1.0))) break;  // invariant subspace: T is exact
        const double ib = 1.0 / bnorm;
        for (int i = tid; i < n; i += SP2_BOUND_THREADS) {
            qp[i] = q[i];
            q[i] = w[i] * ib;
        }
        bprev = bnorm;
        __syncthreads();
    }
    __syncthreads();
    if (warp == 0) {
        // Gershgorin interval of T contains its spectrum
        double tlo = 1e300, thi = -1e300;
        for (int i = 0; i < m; ++i) {
            const double rad = (i > 0 ? fabs(beta[i - 1]) : 0.0) + (i + 1 < m ? fabs(beta[i]) : 0.0);
            tlo = fmin(tlo, alpha[i] - rad);
            thi = fmax(thi, alpha[i] + rad);
        }
        const double pad = 1e-12 * (fabs(tlo) + fabs(thi)) + 1e-300;
        tlo -= pad;
        thi += pad;
        const double th_min = lz_eig_warp(alpha, beta, m, 0, tlo, thi);
        const double th_max = lz_eig_warp(alpha, beta, m, m - 1, tlo, thi);
        if (lane != 0) return;
        const double width = fmax(th_max - th_min, 1e-6);
        const double eps = 1e-8 * (fabs(th_min) + fabs(th_max) + 1.0);
        const double bm = beta[m - 1];
        const double r_min = fabs(bm) * lz_last_component(alpha, beta, m, th_min - eps);
        const double r_max = fabs(bm) * lz_last_component(alpha, beta, m, th_max + eps);
        double lo = th_min - r_min - 0.005 * width;
        double hi = th_max + r_max + 0.005 * width;
        if (!isfinite(lo) || !isfinite(hi) || !(hi > lo)) {
            lo = glo;
            hi = ghi;
        }
        jb.bounds[0] = fmax(lo, glo);
        jb.bounds[1] = fmin(hi, ghi);
        jb.bounds[2] = 0.0;
        jb.bounds[3] = jb.bounds[1] - jb.bounds[0];
    }
}

// The interval from the Lanczos tridiagonal (alpha, beta of m steps) and the Gershgorin bounds.
__device__ void lz_interval(const double* alpha, const double* beta, int m, double glo, double ghi, double* out) {
    double tlo = 1e300, thi = -1e300;
    for (int i = 0; i < m; ++i) {
        const double rad = (i > 0 ? fabs(beta[i - 1]) : 0.0) + (i + 1 < m ? fabs(beta[i]) : 0.0);
        tlo = fmin(tlo, alpha[i] - rad);
        thi = fmax(thi, alpha[i] + rad);
    }
    const double pad = 1e-12 * (fabs(tlo) + fabs(thi)) + 1e-300;
    tlo -= pad;
    thi += pad;
    const double th_min = lz_eig(alpha, beta, m, 0, tlo, thi);
    const double th_max = lz_eig(alpha, beta, m, m - 1, tlo, thi);
    const double width = fmax(th_max - th_min, 1e-6);
    const double eps = 1e-8 * (fabs(th_min) + fabs(th_max) + 1.0);
    const double bm = beta[m - 1];
    const double r_min = fabs(bm) * lz_last_component(alpha, beta, m, th_min - eps);
    const double r_max = fabs(bm) * lz_last_component(alpha, beta, m, th_max + eps);
    double lo = th_min - r_min - 0.005 * width;
    double hi = th_max + r_max + 0.005 * width;
    if (!isfinite(lo) || !isfinite(hi) || !(hi > lo)) {
        lo = glo;
        hi = ghi;
    }
    out[0] = fmax(lo, glo);
    out[1] = fmin(hi, ghi);
}

// k_sp2_bounds for one matrix too large for one CTA (no eigensolver fallback, n > ~448): the same
// Lanczos run by a group of G CTAs, either the whole GPU (one cooperative launch per matrix) or a
// thread-block cluster (one cluster per matrix, all such matrices of a batch in one launch).
// Row r of F* belongs to CTA r % G; the vectors live in global scratch (job.X1, free until
// purification starts) and every CTA keeps the same alpha, beta (sums of the per-CTA shares in one
// fixed order).  Three group barriers per step; cross-CTA data is read through L2 (__ldcg).
// Scratch: q[3][n] | share[2][G].
// Bound by L2 latency: a lane loads LZ_AHEAD elements of two rows before it uses any, and the vector updates take a
// row per lane (14 matrices above 448 orbitals, a cluster each: 394 -> 336 us a launch).
constexpr int LZ_AHEAD = 4;

template <class Sync>
__device__ void sp2_bounds_group(const Sp2Job& jb, int G, int gi, Sync sync) {
    const int n = jb.n;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NW = SP2_BOUND_THREADS / 32;
    double* qb = jb.X1;                 // three Lanczos vectors
    double* share = qb + 3 * (size_t)n; // [2][G]
    __shared__ double red[NW + 2];
    __shared__ double alpha[SP2_LANCZOS], beta[SP2_LANCZOS];
    auto bsum = [&](double v) {
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        __syncthreads();
        if (lane == 0) red[warp] = v;
        __syncthreads();
        double t = 0.0;
        for (int q = 0; q < NW; ++q) t += red[q];
        __syncthreads();
        return t;
    };
    // Gershgorin interval and the start vector (every CTA computes the norm itself)
    double glo = 1e300, ghi = -1e300, nq = 0.0;
    for (int i = tid; i < n; i += SP2_BOUND_THREADS) {
        glo = fmin(glo, jb.rowmin[i]);
        ghi = fmax(ghi, jb.rowmax[i]);
        const double x = cos(0.7 * i + 0.3) + 0.5;
        nq += x * x;
    }
    for (int o = 16; o > 0; o >>= 1) {
        glo = fmin(glo, __shfl_xor_sync(0xffffffffu, glo, o));
        ghi = fmax(ghi, __shfl_xor_sync(0xffffffffu, ghi, o));
    }
    __shared__ double gred[2][NW];
    if (lane == 0) {
        gred[0][warp] = glo;
        gred[1][warp] = ghi;
    }
    nq = bsum(nq);
    glo = gred[0][0];
    ghi = gred[1][0];
    for (int v = 1; v < NW; ++v) {
        glo = fmin(glo, gred[0][v]);
        ghi = fmax(ghi, gred[1][v]);
    }
    const double inq = 1.0 / sqrt(nq);
    for (int i = gi * SP2_BOUND_THREADS + tid; i < n; i += G * SP2_BOUND_THREADS) {
        qb[i] = (cos(0.7 * i + 0.3) + 0.5) * inq;  // q_0
        qb[2 * (size_t)n + i] = 0.0;            // q_{-1}
    }
    sync();
    const int K = min(SP2_LANCZOS, n);
    int m = 0, cur = 0, prv = 2;
    double bprev = 0.0;
    for (int j = 0; j < K; ++j) {
        const int nxt = 3 - cur - prv;  // the third buffer: w, then q_{j+1}
        const double* q = qb + (size_t)cur * n;
        const double* qp = qb + (size_t)prv * n;
        double* wq = qb + (size_t)nxt * n;
        // w_r = F[r, :] . q for own rows (a warp per row) and the CTA's share of q . w
        double part = 0.0;
        for (int r = gi + warp * G; r < n; r += 2 * NW * G) {
            const int r2 = r + NW * G;
            const bool two = r2 < n;  // uniform over the warp
            const double* Fr = jb.F + (long long)r * n;
            const double* Fs = jb.F + (long long)(two ? r2 : r) * n;
            double acc = 0.0, acc2 = 0.0;
            for (int c0 = lane; c0 < n; c0 += 32 * LZ_AHEAD) {
                double x[LZ_AHEAD], y[LZ_AHEAD], v[LZ_AHEAD];
#pragma unroll
                for (int u = 0; u < LZ_AHEAD; ++u) {
                    const int c = c0 + 32 * u;
                    x[u] = c < n ? Fr[c] : 0.0;
                    y[u] = two && c < n ? Fs[c] : 0.0;
                    v[u] = c < n ? __ldcg(q + c) : 0.0;
                }
#pragma unroll
                for (int u = 0; u < LZ_AHEAD; ++u)
                    if (c0 + 32 * u < n) {
                        acc = fma(x[u], v[u], acc);
                        acc2 = fma(y[u], v[u], acc2);
                    }
            }
            for (int o = 16; o > 0; o >>= 1) {
                acc += __shfl_xor_sync(0xffffffffu, acc, o);
                acc2 += __shfl_xor_sync(0xffffffffu, acc2, o);
            }
            if (lane == 0) {
                wq[r] = acc;
                if (two) wq[r2] = acc2;
            }
            part += acc * __ldcg(q + r);
            if (two) part += acc2 * __ldcg(q + r2);
        }
        part = bsum(lane == 0 ? part : 0.0);
        if (tid == 0) share[gi] = part;
        sync();
        const double a = group_share_sum(share, G);
        // w <- w - a q - b_prev q_prev on own rows, the CTA's share of |w|^2
        part = 0.0;
        for (int r0 = gi + warp * G; r0 < n; r0 += 32 * NW * G) {  // a row per lane, summed in row order
            const int r = r0 + lane * NW * G;
            double x = 0.0;
            if (r < n) {
                x = __ldcg(wq + r) - a * __ldcg(q + r) - bprev * __ldcg(qp + r);
                wq[r] = x;
            }
            const int rows = min(32, (n - r0 + NW * G - 1) / (NW * G));
            for (int k = 0; k < rows; ++k) {
                const double xk = __shfl_sync(0xffffffffu, x, k);
                part += xk * xk;
            }
        }
        if (lane != 0) part = 0.0;
        part = bsum(part);
        if (tid == 0) share[G + gi] = part;
        sync();
        const double bnorm = sqrt(group_share_sum(share + G, G));
        if (tid == 0) {
            alpha[j] = a;
            beta[j] = bnorm;
        }
        m = j + 1;
        if (!(bnorm > 1e-12 * fmax(fabs(a), 1.0))) break;  // invariant subspace: T is exact (uniform)
        const double ib = 1.0 / bnorm;
        for (int r = gi + (warp + lane * NW) * G; r < n; r += 32 * NW * G) wq[r] = __ldcg(wq + r) * ib;
        bprev = bnorm;
        prv = cur;
        cur = nxt;
        sync();
    }
    __syncthreads();
    if (gi == 0 && tid == 0) lz_interval(alpha, beta, m, glo, ghi, jb.bounds);
}

__global__ void __launch_bounds__(SP2_BOUND_THREADS, 2) k_sp2_bounds_big(const Sp2Job* __restrict__ jobs, int job,
                                                                       const MolState* __restrict__ st) {
    cg::grid_group grid = cg::this_grid();
    const Sp2Job jb = jobs[job];
    if (!st[jb.mol].active) return;  // uniform over the grid
    sp2_bounds_group(jb, (int)gridDim.x, (int)blockIdx.x, [&] { grid.sync(); });
}

// One cluster (gridDim.x CTAs) per large matrix; blockIdx.y indexes big[], the purification jobs
// without the eigensolver fallback.
__global__ void __launch_bounds__(SP2_BOUND_THREADS, 2) k_sp2_bounds_cl(const Sp2Job* __restrict__ jobs, const int* __restrict__ big,
                                                                      const MolState* __restrict__ st) {
    cg::cluster_group cl = cg::this_cluster();
    const Sp2Job jb = jobs[big[blockIdx.y]];
    if (!st[jb.mol].active) return;  // uniform over the cluster
    sp2_bounds_group(jb, (int)cl.num_blocks(), (int)cl.block_rank(), [&] { cl.sync(); });
}

// X0 = (e_max I - F*) / (e_max - e_min); per-block partial sums of tr X0 and ||X0||_F^2.
__global__ void k_sp2_init(const Sp2Job* __restrict__ jobs, Sp2State* __restrict__ sst, const MolState* __restrict__ st, int nblk) {
    const Sp2Job jb = jobs[blockIdx.y];
    if (!st[jb.mol].active || sp2_fused_now(jb, st[jb.mol].lowp)) return;
    const int n = jb.n;
    const int nb = sp2_init_blocks(n);
    if ((int)blockIdx.x >= nb) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    __shared__ double red[2][32];
    const double emin = jb.bounds[0], emax = jb.bounds[1];  // from k_sp2_bounds
    const double inv = 1.0 / fmax(emax - emin, 1e-300);
    const bool lowp = st[jb.mol].lowp;
    double tr = 0.0, fr = 0.0;
    for (int r = blockIdx.x * nw + warp; r < n; r += nb * nw) {
        const double* Fr = jb.F + (long long)r * n;
        if (lowp) {  // FP32 iterate (rows of ldf floats, pad columns zero in both buffers)
            float* Xr = jb.Xf0 + (long long)r * jb.ldf;
            for (int c = lane; c < jb.ldf; c += 32) {
                const float xf = c < n ? (float)(((c == r ? emax : 0.0) - Fr[c]) * inv) : 0.0f;
                const float x = jb.lowp_tc == 1 ? xf : tf32_round(xf);  // 3xTF32 keeps the full FP32 iterate
                Xr[c] = x;
                if (c >= n) jb.Xf1[(long long)r * jb.ldf + c] = 0.0f;
                fr += (double)x * x;
                if (c == r) tr += x;
            }
            continue;
        }
        double* Xr = jb.X0 + (long long)r * n;
        // four columns per lane per trip, their loads before their stores (each lane keeps its order)
        for (int c0 = lane; c0 < n; c0 += 128) {
            double f[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) f[u] = c0 + 32 * u < n ? Fr[c0 + 32 * u] : 0.0;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int c = c0 + 32 * u;
                if (c >= n) break;
                const double x = ((c == r ? emax : 0.0) - f[u]) * inv;
                Xr[c] = x;
                fr += x * x;
                if (c == r) tr += x;
            }
        }
        if (jb.oz) {  // the digit planes of X0, and zero pad columns in both digit buffers
            const long long plane = (long long)n * jb.ldq;
            for (int c = lane; c < jb.ldq; c += 32) {
                const long long o = (long long)r * jb.ldq + c;
                if (c < n) {
                    oz_digits_of(Xr[c], jb.Dq0, plane, o);
                } else {
                    for (int i = 0; i < kOzPlanes; ++i) jb.Dq0[i * plane + o] = jb.Dq1[i * plane + o] = 0;
                }
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        tr += __shfl_xor_sync(0xffffffffu, tr, o);
        fr += __shfl_xor_sync(0xffffffffu, fr, o);
    }
    if (lane == 0) {
        red[0][warp] = tr;
        red[1][warp] = fr;
    }
    __syncthreads();
    if (tid == 0) {
        double a = 0.0, b = 0.0;
        for (int w = 0; w < nw; ++w) {
            a += red[0][w];
            b += red[1][w];
        }
        jb.part[2 * blockIdx.x] = a;
        jb.part[2 * blockIdx.x + 1] = b;
        if (blockIdx.x == 0) {
            Sp2State& s = sst[blockIdx.y];
            s.emin = emin;
            s.emax = emax;
        }
    }
}

// Sum of `count` (trace, Frobenius) partial pairs in order, by one warp: the lanes fetch 64 pairs at a
// time into the warp's shared buffer (the next 64 in flight meanwhile), then lane 0 adds the traces and
// lane 1 the Frobenius shares, one after the other.  The order, and so every bit, is that of one thread
// walking the list; that walk cost a memory round trip per few pairs (137 us for the 1176 tiles of a
// 3072-orbital matrix, 15 us with the fetches batched; 35 -> 7 us for a batch with 1200 orbitals).  Lane 0
// gets both sums.
constexpr int SP2_SUM_CHUNK = 64;
__device__ __forceinline__ void sp2_sum_parts(const double* __restrict__ part, int count, double* __restrict__ buf, double& tr, double& fr) {
    const int lane = threadIdx.x & 31;
    constexpr int PER = 2 * SP2_SUM_CHUNK / 32;
    double v[PER], t = 0.0;
#pragma unroll
    for (int u = 0; u < PER; ++u) v[u] = lane + 32 * u < 2 * count ? __ldcg(part + lane + 32 * u) : 0.0;
    for (int k0 = 0; k0 < count; k0 += SP2_SUM_CHUNK) {
#pragma unroll
        for (int u = 0; u < PER; ++u) buf[lane + 32 * u] = v[u];
        __syncwarp();
        const int at = 2 * (k0 + SP2_SUM_CHUNK) + lane;
#pragma unroll
        for (int u = 0; u < PER; ++u) v[u] = at + 32 * u < 2 * count ? __ldcg(part + at + 32 * u) : 0.0;
        if (lane < 2) {
            const int m = min(SP2_SUM_CHUNK, count - k0);
            if (m == SP2_SUM_CHUNK) {
#pragma unroll 16
                for (int k = 0; k < SP2_SUM_CHUNK; ++k) t += buf[2 * k + lane];
            } else {
                for (int k = 0; k < m; ++k) t += buf[2 * k + lane];
            }
        }
        __syncwarp();
    }
    tr = t;
    fr = __shfl_sync(0xffffffffu, t, 1);
}

// Reduce the init partials: state of step 0.  A warp per channel.
__global__ void __launch_bounds__(32 * SP2_UPDATE_WARPS) k_sp2_start(const Sp2Job* __restrict__ jobs, Sp2State* __restrict__ sst,
                                                                     const MolState* __restrict__ st, int njobs, int nblk) {
    __shared__ double buf[SP2_UPDATE_WARPS][2 * SP2_SUM_CHUNK];
    const int warp = threadIdx.x >> 5, j = blockIdx.x * SP2_UPDATE_WARPS + warp;
    if (j >= njobs) return;
    const Sp2Job& jb = jobs[j];
    const MolState& ms = st[jb.mol];
    if (sp2_fused_now(jb, ms.lowp)) {
        if ((threadIdx.x & 31) == 0) sst[j].active = 0;
        return;
    }
    double tr, fr;
    sp2_sum_parts(jb.part, sp2_init_blocks(jb.n), buf[warp], tr, fr);
    if ((threadIdx.x & 31) != 0) return;
    Sp2State& s = sst[j];
    s.active = ms.active;
    s.lowp = ms.lowp;
    s.steps = 0;
    s.cur = 0;
    s.converged = 0;
    s.trX = tr;
    s.trX2 = fr;
    s.idem[0] = s.idem[1] = 1e300;
    s.square = fabs(fr - jb.nocc) < fabs(2.0 * tr - fr - jb.nocc) ? 1 : 0;
}

// Epilogue of one purification-step tile: Y = X^2 or 2X - X^2 for r <= c, mirrored; the tile's
// partial trace and Frobenius sums into the job's partials (the job fields it needs are read only
// now, so they hold no registers during the k-loop).
__device__ __forceinline__ void sp2_step_epilogue(const Sp2Job* __restrict__ jp, const Sp2State* __restrict__ sp, int t, int n,
                                                  int m0, int n0, const double acc[2][4][4], bool compute, double red[2][4]) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cur = sp->cur;
    const double* X = cur ? jp->X1 : jp->X0;
    double* Y = cur ? jp->X0 : jp->X1;
    const int square = sp->square;
    double tr = 0.0, fr = 0.0;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int r = m0 + dg_row(i, e);
                const int c = n0 + dg_col(j, e);
                if (compute && r <= c && c < n) {
                    const double x2 = acc[i][j][e];
                    const double y = square ? x2 : 2.0 * X[(long long)r * n + c] - x2;
                    Y[(long long)r * n + c] = y;
                    if (r < c) {
                        Y[(long long)c * n + r] = y;
                        fr += 2.0 * y * y;
                    } else {
                        fr += y * y;
                        tr += y;
                    }
                }
            }
    for (int o = 16; o > 0; o >>= 1) {
        tr += __shfl_xor_sync(0xffffffffu, tr, o);
        fr += __shfl_xor_sync(0xffffffffu, fr, o);
    }
    if (lane == 0) {
        red[0][warp] = tr;
        red[1][warp] = fr;
    }
    __syncthreads();
    if (tid == 0) {
        double* p = jp->part + 2 * (t - jp->tile0);
        p[0] = red[0][0] + red[0][1] + red[0][2] + red[0][3];
        p[1] = red[1][0] + red[1][1] + red[1][2] + red[1][3];
    }
}

// One SP2 step over all upper-triangle 64x64 tiles of every active channel (operands copied by
// cp.async: k_sp2_step8 for odd n, and k_sp2_step16 where the tensor-map kernel is not used).
template <bool PAIRS>
__device__ __forceinline__ void sp2_step_body(const Sp2Job* __restrict__ jobs, const GemmTile* __restrict__ tiles, int t,
                                              const Sp2State* __restrict__ sst, double* dsm, double red[2][4]) {
    const GemmTile tl = tiles[t];
    const Sp2State* sp = sst + tl.job;
    const Sp2Job* jp = jobs + tl.job;
    if (!sp->active || sp->lowp || jp->oz) return;  // TF32 runs: k_sp2_step_tf32 / _tc; digit products: k_sp2_step_oz
    const int n = jp->n;
    const double* X = sp->cur ? jp->X1 : jp->X0;
    const int m0 = tl.tm * DG_TILE, n0 = tl.tn * DG_TILE;
    // only the upper triangle of X^2 is computed: a warp whose quarter is padding or lies below
    // the diagonal of a diagonal tile issues no MMAs
    const bool compute = dg_quarter_on(m0, n0, n, n, tl.tm == tl.tn);
    double acc[2][4][4];
    dg_mainloop<PAIRS>(dsm, X, n, X, n, n, n, n, m0, n0, acc, compute);  // X symmetric: X[rows m0..] . X[:, n0..]
    sp2_step_epilogue(jp, sp, t, n, m0, n0, acc, compute, red);
}

// The same step for even n with the operands copied by the tensor memory accelerator from the
// job's tensor maps (maps[4 job + cur] describes the current iterate), through the mbarrier
// pipeline of dg_mainloop_tma: bit-identical to k_sp2_step16.  A copy wait that runs out sets bit
// 11 of *err and the tile is left unwritten.
__device__ __forceinline__ void sp2_step_tma_body(const Sp2Job* __restrict__ jobs, const GemmTile* __restrict__ tiles, int t,
                                                  const Sp2State* __restrict__ sst, const TmaDesc* __restrict__ maps,
                                                  int* __restrict__ err, unsigned char* dtsm, DtBars& bars, double red[2][4]) {
    const GemmTile tl = tiles[t];
    const Sp2State* sp = sst + tl.job;
    const Sp2Job* jp = jobs + tl.job;
    if (!sp->active || sp->lowp || jp->oz) return;
    const int n = jp->n;
    const int m0 = tl.tm * DG_TILE, n0 = tl.tn * DG_TILE;
    const int shape = dg_quarter_shape(m0, n0, n, n, tl.tm == tl.tn);
    const bool compute = shape != 0;
    const TmaDesc* map = maps + 4 * tl.job + sp->cur;
    double acc[2][4][4];
    if (!dg_mainloop_tma(dt_stages(dtsm), bars, map, map, nullptr, nullptr, tl.tm == tl.tn, n, m0, n0, acc, shape)) {
        if (threadIdx.x == 0) atomicOr(err, 1 << 11);
        return;
    }
    sp2_step_epilogue(jp, sp, t, n, m0, n0, acc, compute, red);
}

__global__ void __launch_bounds__(DG_THREADS, 4) k_sp2_step_tma(const Sp2Job* __restrict__ jobs, const GemmTile* __restrict__ tiles,
                                                               int ntiles, const Sp2State* __restrict__ sst,
                                                               const TmaDesc* __restrict__ maps, int* __restrict__ err) {
    extern __shared__ __align__(16) unsigned char dtsm[];
    __shared__ DtBars bars;
    __shared__ double red[2][4];
    if ((int)blockIdx.x < ntiles) sp2_step_tma_body(jobs, tiles, (int)blockIdx.x, sst, maps, err, dtsm, bars, red);
}

// Both kinds of tiles in one launch: the first nother CTAs take those of odd n, as k_sp2_step8.  Alone these are a
// launch of less than a wave that lasts as long as its largest matrix' k-loop, with the GPU half empty; here
// the even ones fill it (64 molecules of mixed sizes 137 -> 128 ms, 1152 with one radical in nine 163 -> 159).  A kernel of
// its own, since the TMA path takes 7 registers more beside the other (0.4% of a batch of even orders).
__global__ void __launch_bounds__(DG_THREADS, 4) k_sp2_step_both(const Sp2Job* __restrict__ jobs, const GemmTile* __restrict__ tiles,
                                                                int ntiles, const GemmTile* __restrict__ other, int nother,
                                                                const Sp2State* __restrict__ sst,
                                                                const TmaDesc* __restrict__ maps, int* __restrict__ err) {
    extern __shared__ __align__(16) unsigned char dtsm[];
    __shared__ DtBars bars;
    __shared__ double red[2][4];
    const int t = (int)blockIdx.x - nother;
    if (t < 0) sp2_step_body<false>(jobs, other, (int)blockIdx.x, sst, (double*)dtsm, red);
    else if (t < ntiles) sp2_step_tma_body(jobs, tiles, t, sst, maps, err, dtsm, bars, red);
}

// After a step: reduce the tile partials (in tile order), test idempotency, choose the next branch.
// The update of channel j after its product, by one warp (buf: its 2 SP2_SUM_CHUNK doubles of shared
// memory); lane 0 returns true while the channel still purifies.
__device__ __forceinline__ bool sp2_update_job(const Sp2Job* __restrict__ jobs, Sp2State* __restrict__ sst, int j, int max_steps,
                                               double* __restrict__ work, double* __restrict__ buf) {
    Sp2State& s = sst[j];
    if (!s.active) return false;  // uniform over the warp
    const Sp2Job& jb = jobs[j];
    // the partial sums come from the tiles of the kernel that took the product
    const bool lowp = s.lowp != 0;
    const int nparts = lowp ? (jb.lowp_tc ? jb.tc_ntiles : jb.ntiles) : (jb.oz ? jb.oz_ntiles : jb.ntiles);
    double tr, fr;
    sp2_sum_parts(jb.part, nparts, buf, tr, fr);
    __syncwarp();
    if ((threadIdx.x & 31) != 0) return false;
    // algorithmic work of the product just taken: a symmetric X.X, n^3 flops
    const double nd = (double)jb.n;
    if (lowp) {
        atomicAdd(&work[4], 1.0);
        atomicAdd(&work[5], nd * nd * nd);
    } else {
        atomicAdd(&work[0], 1.0);
        atomicAdd(&work[1], nd * nd * nd);
        atomicAdd(&work[3], 16.0 * nd * nd);  // read X, write X^2 (both triangles), FP64
    }
    const double nocc = jb.nocc;
    s.cur ^= 1;
    s.steps += 1;
    s.trX = tr;
    s.trX2 = fr;
    // idempotency error tr X - tr X^2 (sum of x(1-x) over the spectrum, >= 0)
    const double idem = fabs(tr - fr);
    const bool floor_reached = idem < 1.0e-6 && idem >= s.idem[0];  // stagnation at the rounding floor
    // TF32 runs stop at their own rounding level (about 1e-6 relative per eigenvalue), and their
    // result is always taken: it only starts the FP64 iterations
    const bool low_done = lowp && ((idem < 1.0e-2 * jb.n && idem >= s.idem[0]) || idem < 1.0e-5 * jb.n);
    s.idem[0] = s.idem[1];
    s.idem[1] = idem;
    if (low_done || floor_reached || idem < 1.0e-15 * fmax(1.0, nd)) {
        s.active = 0;
        s.converged = 1;
        return false;
    }
    if (s.steps >= max_steps) {
        s.active = 0;
        s.converged = s.lowp;
        return false;
    }
    s.square = fabs(fr - nocc) < fabs(2.0 * tr - fr - nocc) ? 1 : 0;
    return true;
}

__global__ void __launch_bounds__(32 * SP2_UPDATE_WARPS) k_sp2_update(const Sp2Job* __restrict__ jobs, Sp2State* __restrict__ sst,
                                                                      int njobs, int max_steps, int* __restrict__ active_count,
                                                                      double* __restrict__ work) {
    __shared__ double buf[SP2_UPDATE_WARPS][2 * SP2_SUM_CHUNK];
    const int warp = threadIdx.x >> 5, j = blockIdx.x * SP2_UPDATE_WARPS + warp;
    if (j >= njobs) return;
    if (sp2_update_job(jobs, sst, j, max_steps, work, buf[warp])) atomicAdd(active_count, 1);
}

// The update of every channel and the purification loop's decision in one launch (the captured
// solve): the same per-channel update; the last CTA to finish (a ticket in *loop) has the count of
// the channels still purifying and sets the loop's condition.  The tickets and the count start at
// zero (k_sp2_arm) and are put back to zero by that CTA.
__global__ void __launch_bounds__(32 * SP2_UPDATE_WARPS) k_sp2_update_cond(const Sp2Job* __restrict__ jobs, Sp2State* __restrict__ sst,
                                                                           int njobs, int max_steps, double* __restrict__ work,
                                                                           cudaGraphConditionalHandle h, GraphLoop* __restrict__ loop) {
    __shared__ double buf[SP2_UPDATE_WARPS][2 * SP2_SUM_CHUNK];
    const int warp = threadIdx.x >> 5, j = blockIdx.x * SP2_UPDATE_WARPS + warp;
    const bool more_j = j < njobs && sp2_update_job(jobs, sst, j, max_steps, work, buf[warp]);
    const int more = __syncthreads_count(more_j);
    if (threadIdx.x != 0) return;
    int active = more;
    if (gridDim.x > 1) {
        if (more) atomicAdd(&loop->sp2_active, more);
        __threadfence();
        if (atomicAdd(&loop->ticket, 1) != (int)gridDim.x - 1) return;
        __threadfence();
        active = atomicExch(&loop->sp2_active, 0);
        loop->ticket = 0;
    }
    const int step = loop->sp2_step + 1;
    loop->sp2_step = step;
    loop->sp2_total += 1;
    cudaGraphSetConditional(h, (active > 0 && step < max_steps) ? 1u : 0u);
}

// P_new = w X (the converged X); molecules whose purification stalled are flagged for the
// eigensolver path: need_eigen (cluster Jacobi, up to 448 orbitals) or big_stall per channel job
// and the count in big_count (the large-matrix eigensolver, above 448).
__global__ void k_sp2_finish(const Sp2Job* __restrict__ jobs, const Sp2State* __restrict__ sst, const MolState* __restrict__ st,
                             int* __restrict__ need_eigen, double* __restrict__ work, int* __restrict__ big_stall,
                             int* __restrict__ big_count) {
    const Sp2Job jb = jobs[blockIdx.y];
    if (!st[jb.mol].active || sp2_fused_now(jb, st[jb.mol].lowp)) return;
    const Sp2State& s = sst[blockIdx.y];
    if (!s.converged) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            atomicAdd(&work[2], 1.0);
            if (jb.fallback) {
                need_eigen[jb.mol] = need_eigen[-1] = 1;
            } else {  // above the cluster Jacobi's size: the host runs the large-matrix eigensolver
                big_stall[blockIdx.y] = 1;
                atomicAdd(big_count, 1);
            }
        }
        return;
    }
    const long long nn = (long long)jb.n * jb.n;
    if (s.lowp) {
        // the TF32 iterate, rescaled to the exact electron count (its trace is off by the rounding)
        const float* Xf = s.cur ? jb.Xf1 : jb.Xf0;
        const double w = jb.weight * (s.trX > 0.0 ? jb.nocc / s.trX : 1.0);
        for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += (long long)gridDim.x * blockDim.x) {
            const long long r = i / jb.n, c = i - r * jb.n;
            jb.P[i] = w * (double)Xf[r * jb.ldf + c];
        }
        return;
    }
    const double* X = s.cur ? jb.X1 : jb.X0;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x; i0 < nn; i0 += 4 * stride) {
        double x[4];  // P may be X0: every load of the trip before its stores
#pragma unroll
        for (int u = 0; u < 4; ++u) x[u] = i0 + u * stride < nn ? X[i0 + u * stride] : 0.0;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i0 + u * stride < nn) jb.P[i0 + u * stride] = jb.weight * x[u];
    }
}

size_t dgemm_smem_bytes() { return DG_SMEM; }
size_t dgemm_tma_smem_bytes() { return DT_SMEM; }
size_t dgemm_both_smem_bytes() { return DG_SMEM > DT_SMEM ? DG_SMEM : DT_SMEM; }  // four CTAs still fit an SM

__global__ void __launch_bounds__(DG_THREADS, 4) k_sp2_step16(const Sp2Job* __restrict__ jobs, const GemmTile* __restrict__ tiles,
                                                              int ntiles, const Sp2State* __restrict__ sst) {
    extern __shared__ __align__(16) double dsm[];
    __shared__ double red[2][4];
    if ((int)blockIdx.x < ntiles) sp2_step_body<true>(jobs, tiles, (int)blockIdx.x, sst, dsm, red);
}
__global__ void __launch_bounds__(DG_THREADS, 4) k_sp2_step8(const Sp2Job* __restrict__ jobs, const GemmTile* __restrict__ tiles,
                                                             int ntiles, const Sp2State* __restrict__ sst) {
    extern __shared__ __align__(16) double dsm[];
    __shared__ double red[2][4];
    if ((int)blockIdx.x < ntiles) sp2_step_body<false>(jobs, tiles, (int)blockIdx.x, sst, dsm, red);
}

}  // namespace am1
