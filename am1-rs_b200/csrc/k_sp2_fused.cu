// A whole purification (spectral bounds, start, every product, the stop, P) of one channel in one launch.
//
// The launch-per-step form (k_sp2.cu) fills the GPU when a batch has thousands of tiles.  A lone molecule, or
// a small matrix anywhere, is bound by latency there: a product of a few microseconds, an update of as
// many, and the gaps between launches, 12 to 20 times per SCF iteration.  Here the loop stays on chip:
//   k_sp2_res  one CTA per matrix of up to FU_RES_MAX orbitals, both iterates in shared memory
//   k_sp2_clu  one cluster per matrix of up to FU_CLU_MAX orbitals, the iterates in L2 (scratch rows padded to 32),
//              32-row panels fetched by cp.async; one cluster barrier per product
// The products are DMMA m16n8k8 blocks over ascending k, and every sum (Lanczos dots, start, tile sums) is
// taken in the order of the launch-per-step kernels, whose unit is the 32 x 32 quarter of a 64 x 64 tile,
// so the density is bit-identical and the choice of kernel is only a choice of speed.
// Bound, from clock stamps inside the kernels (cycles per product): res by the DMMA pipe of its SM from 64 orbitals
// on (n = 112: 17.2k in the products, whose MMAs alone are 12.5k, 3.3k in the sums and the update; n = 8: 0.9k
// and 1.6k); clu by the L2 reads of the one GPC its cluster lies in (n = 192: 11.6k for 6.1k of MMAs, 1.6k in
// the cluster barrier, sums and update).  Behind a Lanczos run (the first SCF iterations) the Ritz values cost
// another 41k, 129 cycles to a division.  Measured, launch per step -> one launch: methane (8 orbitals) 2.54 ->
// 1.14 ms a solve, C13H27 (79) 7.60 -> 4.07, 32 waters (192) 7.49 -> 4.09, a 384-orbital purification alone 1.39 ->
// 1.12.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "am1gpu_internal.h"
#include "dmma_gemm.cuh"
#include "kernels.h"
#include "sp2_lanczos.cuh"

namespace am1 {

namespace cg = cooperative_groups;

constexpr int FU_THREADS = 256, FU_WARPS = FU_THREADS / 32;
constexpr int FU_VW = 8;          // warps per block of k_sp2_init, whose partial sums are reproduced
constexpr int FU_KC = 32;         // columns of a panel chunk
constexpr int FU_LD = FU_KC + 4;  // its row stride in shared memory (conflict-free fragment loads)
constexpr int FU_STAGES = 4, FU_PANEL = 32 * FU_LD, FU_STAGE = 2 * FU_PANEL;  // per group of four warps: rows R and columns C
constexpr int FU_GROUPS = FU_WARPS / 4;

__host__ __device__ constexpr int fu_tiles(int n) { return (n + 63) / 64 * ((n + 63) / 64 + 1) / 2; }
static_assert(FU_RES_MAX <= FU_CLU_MAX && fu_tiles(FU_CLU_MAX) <= 32, "a lane per tile in the update");
__host__ __device__ inline int fu_res_ld(int n) { return ((n + 7) & ~7) + 4; }
__host__ __device__ inline int fu_clu_ld(int n) { return (n + FU_KC - 1) / FU_KC * FU_KC; }
// doubles of the two scratch iterates of a k_sp2_clu channel: rows padded to 32, columns to whole chunks
long long sp2_clu_doubles(int n) { return 2LL * ((n + 31) & ~31) * fu_clu_ld(n); }

// Dynamic shared memory, in doubles: four vectors, the start's partials, the quarter sums (two buffers),
// then the iterates (res) or the panel stages (clu).
struct FuLayout {
    int vec, init, qsum, main, total;
    __host__ __device__ FuLayout(int n, bool res) {
        const int nv = (n + 1) & ~1;
        vec = 0;
        init = 4 * nv;
        qsum = init + 2 * 32 * FU_VW;
        main = qsum + 2 * 8 * fu_tiles(n);
        total = main + (res ? 2 * ((n + 15) & ~15) * fu_res_ld(n) : FU_GROUPS * FU_STAGES * FU_STAGE);
    }
};
size_t sp2_fused_smem_bytes(int n, bool res) { return sizeof(double) * (size_t)FuLayout(n, res).total; }

// quarter (R, C) of the upper triangle (32-row units) -> its slot: 4 tile + 2 (row half) + column half
__device__ __forceinline__ int fu_slot(int R, int C, int tn) {
    const int x = R >> 1, y = C >> 1;
    return 4 * (x * tn - x * (x - 1) / 2 + (y - x)) + 2 * (R & 1) + (C & 1);
}

__device__ __forceinline__ void fu_butterfly(double& a, double& b) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
}

// Element (r, c) = y of an iterate into its trace and Frobenius sums, without a branch (y is zero outside
// the upper triangle and the matrix, and adding +0 changes no bit): the off-diagonal counts twice.
__device__ __forceinline__ void fu_sum(double y, int r, int c, double& tr, double& fr) {
    fr = fma(r == c ? y : 2.0 * y, y, fr);
    tr += r == c ? y : 0.0;
}

// acc += rows . columns^T over `kn` k-steps of 8, the rows at pa and pa + 8 ld, the columns at pb (and pb + 8 ld
// when TWO), all read along k: the next step's fragments are fetched before this step's MMAs.
template <bool TWO>
__device__ __forceinline__ void fu_kloop(const double* pa, const double* pb, int ld, int kn, double acc[2][4]) {
    double a[4], b[4];
    auto fetch = [&](int k, double (&x)[4], double (&y)[4]) {
        x[0] = pa[k];
        x[1] = pa[k + 8 * ld];
        x[2] = pa[k + 4];
        x[3] = pa[k + 8 * ld + 4];
        y[0] = pb[k];
        y[1] = pb[k + 4];
        if (TWO) {
            y[2] = pb[k + 8 * ld];
            y[3] = pb[k + 8 * ld + 4];
        }
    };
    fetch(0, a, b);
#pragma unroll 2
    for (int k = 1; k < kn; ++k) {
        double an[4], bn[4];
        fetch(8 * k, an, bn);
        dg_mma(acc[0], a, b);
        if (TWO) dg_mma(acc[1], a, b + 2);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            a[u] = an[u];
            b[u] = bn[u];
        }
    }
    dg_mma(acc[0], a, b);
    if (TWO) dg_mma(acc[1], a, b + 2);
}

template <bool RES>
__device__ __forceinline__ void sp2_fused_body(const Sp2Job* __restrict__ jobs, const int* __restrict__ list, Sp2State* __restrict__ sst,
                                               const MolState* __restrict__ st, int* __restrict__ need_eigen, double* __restrict__ work,
                                               int max_steps) {
    extern __shared__ __align__(16) double fsm[];
    __shared__ double red[16], gred[2][FU_WARPS], alpha[SP2_LANCZOS], beta[SP2_LANCZOS], ritz[2], comp[2];
    __shared__ double chain[FU_GROUPS][32][2];
    __shared__ unsigned short item[128];  // res: 16 x 16 sub-blocks; clu: quarters (R, C)
    static_assert((FU_CLU_MAX + 31) / 32 * ((FU_CLU_MAX + 31) / 32 + 1) / 2 <= 128, "item holds every quarter");
    __shared__ int nitem;
    int C = 1, crank = 0;
    if constexpr (!RES) {
        cg::cluster_group cl = cg::this_cluster();
        C = (int)cl.num_blocks();
        crank = (int)cl.block_rank();
    }
    const int job = list[RES ? blockIdx.x : blockIdx.y];
    const Sp2Job& jb = jobs[job];
    const MolState& ms = st[jb.mol];
    if (!ms.active || ms.lowp) return;  // uniform over the cluster
    const int n = jb.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gw = crank * FU_WARPS + warp, ngw = C * FU_WARPS;  // warps of the cluster
    const FuLayout lay(n, RES);
    const int nv = (n + 1) & ~1;
    double* q = fsm;
    double* qp = fsm + nv;
    double* ip = fsm + lay.init;
    double* qsum = fsm + lay.qsum;
    const int tn = (n + 63) / 64, ntiles = fu_tiles(n), nq = (n + 31) / 32;
    auto csync = [&] {
        if constexpr (RES) __syncthreads();
        else cg::this_cluster().sync();
    };
    // the same shared-memory word in CTA `rank` of the cluster
    auto peer = [&](double* p, int rank) -> double* {
        if constexpr (RES) return p;
        else return cg::this_cluster().map_shared_rank(p, rank);
    };
    // sum over the CTA of elements tid (v0) and tid + 256 (v1): the order of k_sp2_bounds' 512 threads
    auto bsum = [&](double v0, double v1) {
        fu_butterfly(v0, v1);
        __syncthreads();
        if (lane == 0) {
            red[warp] = v0;
            red[warp + FU_WARPS] = v1;
        }
        __syncthreads();
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < 16; ++w) t += red[w];
        return t;
    };

    // ---- work lists and Gershgorin interval
    if (tid == 0) {
        int k = 0;
        if constexpr (RES) {
            for (int R = 0; R < nq; ++R)
                for (int Cq = R; Cq < nq; ++Cq)
                    for (int sub = 0; sub < 4; ++sub) {
                        const int r0 = 32 * R + 16 * (sub >> 1), c0 = 32 * Cq + 16 * (sub & 1);
                        if (r0 < n && c0 < n && r0 <= c0) item[k++] = (unsigned short)((r0 >> 4) * 32 + (c0 >> 4));
                    }
        } else {  // off-diagonal quarters first: the diagonal ones issue fewer MMAs
            for (int R = 0; R < nq; ++R)
                for (int Cq = R + 1; Cq < nq; ++Cq) item[k++] = (unsigned short)(R * 32 + Cq);
            for (int R = 0; R < nq; ++R) item[k++] = (unsigned short)(R * 33);
        }
        nitem = k;
    }
    for (int i = tid; i < 2 * 8 * ntiles; i += FU_THREADS) qsum[i] = 0.0;
    double glo = 1e300, ghi = -1e300;
    for (int i = tid; i < n; i += FU_THREADS) {
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
    const size_t xsz = (size_t)(RES ? (n + 15) & ~15 : 32 * nq) * (RES ? fu_res_ld(n) : fu_clu_ld(n));  // one iterate
    double* xb0 = RES ? fsm + lay.main : jb.Xc;
    const double* F = jb.F;
    if constexpr (RES) {  // F* into the second iterate's room (free until the first product)
        double* Fs = xb0 + xsz;
        const double* Fg = jb.F;
        for (int i = tid; i < n * n; i += FU_THREADS) Fs[i] = Fg[i];
        for (int i = tid; i < (int)xsz; i += FU_THREADS) xb0[i] = 0.0;
        F = Fs;
    }
    // ---- the spectral interval (k_sp2_bounds: the previous interval widened, or a Lanczos run)
    const bool may_reuse = jb.rowdf != nullptr && ms.iter > 0;
    const double b_lo = jb.bounds[0], b_hi = jb.bounds[1], b_slack = jb.bounds[2], b_width = jb.bounds[3];
    const double dsum = bsum(may_reuse && tid < n ? jb.rowdf[tid] : 0.0,
                             may_reuse && tid + FU_THREADS < n ? jb.rowdf[tid + FU_THREADS] : 0.0);  // its barriers also publish gred
    glo = gred[0][0];
    ghi = gred[1][0];
    for (int v = 1; v < FU_WARPS; ++v) {
        glo = fmin(glo, gred[0][v]);
        ghi = fmax(ghi, gred[1][v]);
    }
    csync();  // every CTA runs and has read the previous interval
    double emin = 0.0, emax = 0.0;
    bool have = false;
    if (may_reuse) {
        const double delta = sqrt(dsum) * (1.0 + 1e-12);
        const double slack = b_slack + delta;
        const double lo = fmax(b_lo - delta, glo), hi = fmin(b_hi + delta, ghi);
        if (isfinite(slack) && b_width > 0.0 && slack <= SP2_REUSE_FRAC * b_width && hi > lo) {
            have = true;
            emin = lo;
            emax = hi;
            if (crank == 0 && tid == 0) {
                jb.bounds[0] = lo;
                jb.bounds[1] = hi;
                jb.bounds[2] = slack;
            }
        }
    }
    if (!have) {  // uniform over the cluster
        double x0 = 0.0, x1 = 0.0;
        if (tid < n) {
            const int i = tid;
            x0 = cos(0.7 * i + 0.3) + 0.5;
            q[i] = x0;
            qp[i] = 0.0;
        }
        if (tid + FU_THREADS < n) {
            const int i = tid + FU_THREADS;
            x1 = cos(0.7 * i + 0.3) + 0.5;
            q[i] = x1;
            qp[i] = 0.0;
        }
        const double inq = 1.0 / sqrt(bsum(__dmul_rn(x0, x0), __dmul_rn(x1, x1)));
        for (int i = tid; i < n; i += FU_THREADS) q[i] *= inq;
        __syncthreads();
        const int K = min(SP2_LANCZOS, n);
        const bool pairs = (n & 1) == 0 && (reinterpret_cast<uintptr_t>(jb.F) & 15) == 0;
        const int sub = lane >> 3, sl = lane & 7;
        int m = 0;
        double bprev = 0.0;
        for (int j = 0; j < K; ++j) {
            double* w = fsm + (2 + (j & 1)) * nv;  // a CTA one step ahead writes the other buffer
            for (int r0 = 4 * gw; r0 < n; r0 += 4 * ngw) {
                const int r = r0 + sub;
                double acc = 0.0;
                if (r < n) {
                    const double* Fr = F + (long long)r * n;
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
#pragma unroll 4
                        for (int c = sl; c < n; c += 8) acc = fma(Fr[c], q[c], acc);
                    }
                }
                for (int o = 4; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
                if (r < n)
                    for (int k = sl; k < C; k += 8) peer(w, k)[r] = acc;
            }
            csync();
            const int i0 = tid, i1 = tid + FU_THREADS;
            const double a = bsum(i0 < n ? __dmul_rn(q[i0], w[i0]) : 0.0, i1 < n ? __dmul_rn(q[i1], w[i1]) : 0.0);
            double y0 = 0.0, y1 = 0.0;
            if (i0 < n) y0 = w[i0] - a * q[i0] - bprev * qp[i0];
            if (i1 < n) y1 = w[i1] - a * q[i1] - bprev * qp[i1];
            const double bnorm = sqrt(bsum(__dmul_rn(y0, y0), __dmul_rn(y1, y1)));
            if (tid == 0) {
                alpha[j] = a;
                beta[j] = bnorm;
            }
            m = j + 1;
            if (!(bnorm > 1e-12 * fmax(fabs(a), 1.0))) break;  // invariant subspace: T is exact
            const double ib = 1.0 / bnorm;
            if (i0 < n) {
                qp[i0] = q[i0];
                q[i0] = y0 * ib;
            }
            if (i1 < n) {
                qp[i1] = q[i1];
                q[i1] = y1 * ib;
            }
            bprev = bnorm;
            __syncthreads();
        }
        __syncthreads();
        // the extreme Ritz values and their residuals: the lower end on warp 0, the upper on warp 1
        double tlo = 1e300, thi = -1e300;
        for (int i = 0; i < m; ++i) {
            const double rad = (i > 0 ? fabs(beta[i - 1]) : 0.0) + (i + 1 < m ? fabs(beta[i]) : 0.0);
            tlo = fmin(tlo, alpha[i] - rad);
            thi = fmax(thi, alpha[i] + rad);
        }
        const double pad = 1e-12 * (fabs(tlo) + fabs(thi)) + 1e-300;
        tlo -= pad;
        thi += pad;
        if (warp < 2) {
            const double th = lz_eig_warp(alpha, beta, m, warp == 0 ? 0 : m - 1, tlo, thi);
            if (lane == 0) ritz[warp] = th;
        }
        __syncthreads();
        const double th_min = ritz[0], th_max = ritz[1];
        const double width = fmax(th_max - th_min, 1e-6);
        const double eps = 1e-8 * (fabs(th_min) + fabs(th_max) + 1.0);
        if (warp < 2 && lane == 0) comp[warp] = lz_last_component(alpha, beta, m, warp == 0 ? th_min - eps : th_max + eps);
        __syncthreads();
        const double bm = beta[m - 1];
        const double r_min = fabs(bm) * comp[0];
        const double r_max = fabs(bm) * comp[1];
        double lo = th_min - r_min - 0.005 * width;
        double hi = th_max + r_max + 0.005 * width;
        if (!isfinite(lo) || !isfinite(hi) || !(hi > lo)) {
            lo = glo;
            hi = ghi;
        }
        emin = fmax(lo, glo);
        emax = fmin(hi, ghi);
        if (crank == 0 && tid == 0) {
            jb.bounds[0] = emin;
            jb.bounds[1] = emax;
            jb.bounds[2] = 0.0;
            jb.bounds[3] = emax - emin;
        }
    }

    // ---- X0 = (e_max I - F*) / (e_max - e_min), and its trace and Frobenius norm by the warps of k_sp2_init
    const double inv = 1.0 / fmax(emax - emin, 1e-300);
    const int nb = sp2_init_blocks(n);
    const int ld = RES ? fu_res_ld(n) : fu_clu_ld(n);
    if constexpr (!RES) {
        for (int r = gw; r < 32 * nq; r += ngw)  // the pads of both iterates
            for (int c = (r < n ? n : 0) + lane; c < ld; c += 32) xb0[(size_t)r * ld + c] = xb0[xsz + (size_t)r * ld + c] = 0.0;
    }
    for (int vw = gw; vw < nb * FU_VW; vw += ngw) {
        double tr = 0.0, fr = 0.0;
        for (int r = vw; r < n; r += nb * FU_VW) {
            const double* Fr = F + (long long)r * n;
            double* Xr = xb0 + (size_t)r * ld;
#pragma unroll 4
            for (int c = lane; c < n; c += 32) {
                const double x = ((c == r ? emax : 0.0) - Fr[c]) * inv;
                Xr[c] = x;
                fr += x * x;
                if (c == r) tr += x;
            }
        }
        fu_butterfly(tr, fr);
        if (lane < C) {
            peer(ip, lane)[2 * vw] = tr;
            peer(ip, lane)[2 * vw + 1] = fr;
        }
    }
    csync();
    if constexpr (RES) {
        for (int i = tid; i < (int)xsz; i += FU_THREADS) xb0[xsz + i] = 0.0;
        __syncthreads();
    }
    double trX = 0.0, frX = 0.0;
    {
        double a = 0.0, b = 0.0;
        if (lane < nb)
            for (int w = 0; w < FU_VW; ++w) {
                a += ip[2 * (FU_VW * lane + w)];
                b += ip[2 * (FU_VW * lane + w) + 1];
            }
        for (int k = 0; k < nb; ++k) {
            trX += __shfl_sync(0xffffffffu, a, k);
            frX += __shfl_sync(0xffffffffu, b, k);
        }
    }
    const double nocc = jb.nocc, nd = (double)n;
    int square = fabs(frX - nocc) < fabs(2.0 * trX - frX - nocc) ? 1 : 0;
    double idem0 = 1e300, idem1 = 1e300;
    int cur = 0, steps = 0;
    bool converged = false;
    const int g = lane >> 2, tq = lane & 3;
    const int ks = (n + 7) / 8;  // k-steps of 8

    for (;;) {
        const double* X = xb0 + cur * xsz;
        double* Y = xb0 + (cur ^ 1) * xsz;
        double* qs = qsum + (steps & 1) * 8 * ntiles;
        if constexpr (RES) {
            for (int it = warp; it < nitem; it += FU_WARPS) {
                const int r0 = (item[it] >> 5) << 4, c0 = (item[it] & 31) << 4;
                const bool two = c0 + 8 < n;  // the second 8 columns reach the matrix
                const double* xa = X + (r0 + g) * ld + tq;
                const double* xb = X + (c0 + g) * ld + tq;
                double acc[2][4] = {};
                if (two) fu_kloop<true>(xa, xb, ld, ks, acc);
                else fu_kloop<false>(xa, xb, ld, ks, acc);
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int r = r0 + g + (e >= 2 ? 8 : 0), c = c0 + 8 * j + 2 * tq + (e & 1);
                        if (r <= c && c < n) {
                            const double x2 = acc[j][e];
                            const double y = square ? x2 : 2.0 * X[r * ld + c] - x2;
                            Y[r * ld + c] = y;
                            Y[c * ld + r] = y;
                        }
                    }
            }
            __syncthreads();
            // a quarter's sums by one warp, each lane in the order of the tile epilogue (i, j, e)
            for (int p = warp; p < nq * (nq + 1) / 2; p += FU_WARPS) {
                int R = 0, rem = p;
                while (rem >= nq - R) rem -= nq - R++;
                const int Cq = R + rem;
                double tr = 0.0, fr = 0.0;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    double y[16];
#pragma unroll
                    for (int u = 0; u < 16; ++u) {
                        const int e = u & 3, j = u >> 2;
                        const int r = 32 * R + 16 * i + g + (e >= 2 ? 8 : 0), c = 32 * Cq + 8 * j + 2 * tq + (e & 1);
                        y[u] = r <= c && c < n ? Y[r * ld + c] : 0.0;
                    }
#pragma unroll
                    for (int u = 0; u < 16; ++u) {
                        const int e = u & 3, j = u >> 2;
                        const int r = 32 * R + 16 * i + g + (e >= 2 ? 8 : 0), c = 32 * Cq + 8 * j + 2 * tq + (e & 1);
                        fu_sum(y[u], r, c, tr, fr);
                    }
                }
                fu_butterfly(tr, fr);
                if (lane == 0) {
                    const int s = fu_slot(R, Cq, tn);
                    qs[2 * s] = tr;
                    qs[2 * s + 1] = fr;
                }
            }
            __syncthreads();
        } else {
            // Groups of four warps, each with its own quarters, copies and barrier, so one group's fragment loads
            // run under the other's MMAs (the whole CTA in step on chunks shared by two quarters: 20% slower at n =
            // 192).  Quarters go round the CTAs first.  A group walks (quarter, 32-column chunk) in order, the
            // copies FU_STAGES - 1 chunks ahead; chunks of 64 in two stages were 3-6% slower from n = 384 on.
            const int grp = warp >> 2, gid = grp * C + crank, gstep = FU_GROUPS * C, gt = tid & 127;
            double* stg = fsm + lay.main + grp * FU_STAGES * FU_STAGE;
            const int lrow = gt >> 4, lcol = (gt & 15) * 2;
            const double* lsrc = X + (size_t)lrow * ld + lcol;
            double* ldst = stg + lrow * FU_LD + lcol;
            const int nkc = ld / FU_KC;
            int pr = gid, pk = 0, pst = 0;  // next quarter, chunk and stage to copy
            auto issue = [&] {
                if (pr < nitem) {
                    const int R = item[pr] >> 5, Cq = item[pr] & 31;
                    double* dst = ldst + pst * FU_STAGE;
#pragma unroll
                    for (int p = 0; p < 2; ++p) {
                        if (p == 1 && Cq == R) continue;  // a diagonal quarter reads panel 0 twice
                        const double* src = lsrc + (size_t)(32 * (p == 0 ? R : Cq)) * ld + FU_KC * pk;
#pragma unroll
                        for (int u = 0; u < 4; ++u) dg_cp16(dst + p * FU_PANEL + 8 * u * FU_LD, src + (size_t)(8 * u) * ld, X, true);
                    }
                    if (++pk == nkc) {
                        pk = 0;
                        pr += gstep;
                    }
                }
                pst = pst + 1 == FU_STAGES ? 0 : pst + 1;
                dg_commit();
            };
#pragma unroll
            for (int t = 0; t < FU_STAGES - 1; ++t) issue();
            const int i = (warp >> 1) & 1, jh = warp & 1;
            auto gsync = [&] { asm volatile("bar.sync %0, 128;\n" ::"r"(1 + grp) : "memory"); };
            double acc[2][4], xs[2][4];
            int cst = 0;
            for (int cr = gid; cr < nitem; cr += gstep) {
                const int R = item[cr] >> 5, Cq = item[cr] & 31;
                const int r0 = 32 * R + 16 * i, c0 = 32 * Cq + 16 * jh;
                const bool on = r0 < n && c0 < n && r0 <= c0;
                const double* fa = stg + (16 * i + g) * FU_LD + tq;
                const double* fb = stg + (Cq == R ? 0 : FU_PANEL) + (16 * jh + g) * FU_LD + tq;
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[j][e] = 0.0;
                for (int kc = 0; kc < nkc; ++kc) {
                    dg_wait<FU_STAGES - 2>();
                    gsync();
                    issue();
                    if (on) {
                        const double* pa = fa + cst * FU_STAGE;
                        const double* pb = fb + cst * FU_STAGE;
                        const int kn = min(FU_KC / 8, ks - kc * (FU_KC / 8));
                        if (c0 + 8 < n) fu_kloop<true>(pa, pb, FU_LD, kn, acc);
                        else fu_kloop<false>(pa, pb, FU_LD, kn, acc);  // the second 8 columns lie past the matrix
                        if (kc == Cq * 32 / FU_KC) {  // this chunk holds X's own elements of the block
                            const double* P0 = stg + cst * FU_STAGE + (Cq * 32) % FU_KC;
#pragma unroll
                            for (int j = 0; j < 2; ++j)
#pragma unroll
                                for (int e = 0; e < 4; ++e)
                                    xs[j][e] = P0[(16 * i + g + (e >= 2 ? 8 : 0)) * FU_LD + 16 * jh + 8 * j + 2 * tq + (e & 1)];
                        }
                    }
                    cst = cst + 1 == FU_STAGES ? 0 : cst + 1;
                }
                // epilogue of the quarter: Y and its mirror; the quarter's sums pass through its four warps in
                // the tile epilogue's order (row half, then columns)
                double y[2][4];
                if (on) {
#pragma unroll
                    for (int j = 0; j < 2; ++j)
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const int r = r0 + g + (e >= 2 ? 8 : 0), c = c0 + 8 * j + 2 * tq + (e & 1);
                            y[j][e] = 0.0;
                            if (r <= c && c < n) {
                                const double x2 = acc[j][e];
                                y[j][e] = square ? x2 : 2.0 * xs[j][e] - x2;
                                Y[(size_t)r * ld + c] = y[j][e];
                                if (r < c) Y[(size_t)c * ld + r] = y[j][e];
                            }
                        }
                }
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    if ((warp & 3) == p) {
                        double tr = p == 0 ? 0.0 : chain[grp][lane][0], fr = p == 0 ? 0.0 : chain[grp][lane][1];
                        if (on) {
#pragma unroll
                            for (int j = 0; j < 2; ++j)
#pragma unroll
                                for (int e = 0; e < 4; ++e) {
                                    const int r = r0 + g + (e >= 2 ? 8 : 0), c = c0 + 8 * j + 2 * tq + (e & 1);
                                    fu_sum(y[j][e], r, c, tr, fr);
                                }
                        }
                        if (p < 3) {
                            chain[grp][lane][0] = tr;
                            chain[grp][lane][1] = fr;
                        } else {
                            fu_butterfly(tr, fr);
                            const int s = fu_slot(R, Cq, tn);
                            if (lane < C) {
                                peer(qs, lane)[2 * s] = tr;
                                peer(qs, lane)[2 * s + 1] = fr;
                            }
                        }
                    }
                    if (p < 3) gsync();
                }
            }
            csync();  // Y and every quarter's sums are visible to the cluster
        }
        // ---- the update (sp2_update_job): tile sums in tile order, the stop, the next branch
        double tr = 0.0, fr = 0.0;
        {
            double a = 0.0, b = 0.0;
            if (lane < ntiles) {
                const double* p = qs + 8 * lane;
                a = p[0] + p[2] + p[4] + p[6];
                b = p[1] + p[3] + p[5] + p[7];
            }
            for (int t = 0; t < ntiles; ++t) {
                tr += __shfl_sync(0xffffffffu, a, t);
                fr += __shfl_sync(0xffffffffu, b, t);
            }
        }
        cur ^= 1;
        steps += 1;
        const double idem = fabs(tr - fr);
        const bool floor_reached = idem < 1.0e-6 && idem >= idem0;
        idem0 = idem1;
        idem1 = idem;
        if (floor_reached || idem < 1.0e-15 * fmax(1.0, nd)) {
            converged = true;
            break;
        }
        if (steps >= max_steps) break;
        square = fabs(fr - nocc) < fabs(2.0 * tr - fr - nocc) ? 1 : 0;
    }

    // ---- P = w X, or the stall flag; the work counters and the channel's state
    if (converged) {
        const double* X = xb0 + cur * xsz;
        const double weight = jb.weight;
        for (int r = gw; r < n; r += ngw)
#pragma unroll 4
            for (int c = lane; c < n; c += 32)
                jb.P[(long long)r * n + c] = weight * (RES ? X[(size_t)r * ld + c] : __ldcg(X + (size_t)r * ld + c));
    }
    if (crank == 0 && tid == 0) {
        atomicAdd(&work[0], (double)steps);
        atomicAdd(&work[1], (double)steps * nd * nd * nd);
        atomicAdd(&work[3], (double)steps * 16.0 * nd * nd);
        if (!converged) {
            atomicAdd(&work[2], 1.0);
            need_eigen[jb.mol] = need_eigen[-1] = 1;
        }
        Sp2State& s = sst[job];
        s.active = 0;
        s.lowp = 0;
        s.steps = steps;
        s.cur = cur;
        s.converged = converged ? 1 : 0;
    }
    if constexpr (!RES) csync();  // no CTA leaves while another may still address its shared memory
}

__global__ void __launch_bounds__(FU_THREADS, 2) k_sp2_res(const Sp2Job* __restrict__ jobs, const int* __restrict__ list,
                                                           Sp2State* __restrict__ sst, const MolState* __restrict__ st,
                                                           int* __restrict__ need_eigen, double* __restrict__ work, int max_steps) {
    sp2_fused_body<true>(jobs, list, sst, st, need_eigen, work, max_steps);
}

__global__ void __launch_bounds__(FU_THREADS, 1) k_sp2_clu(const Sp2Job* __restrict__ jobs, const int* __restrict__ list,
                                                           Sp2State* __restrict__ sst, const MolState* __restrict__ st,
                                                           int* __restrict__ need_eigen, double* __restrict__ work, int max_steps) {
    sp2_fused_body<false>(jobs, list, sst, st, need_eigen, work, max_steps);
}

}  // namespace am1
