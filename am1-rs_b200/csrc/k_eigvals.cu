// Eigenvalues of the last extrapolated Fock matrix (the reference's mo_energies are the
// eigenvalues of the F* of its last iteration, src/scf.rs:654-689), without eigenvectors:
//   k_tridiag : Householder reduction A = Q T Q^T (Golub & Van Loan, Alg. 8.3.1), the matrix held
//               in the shared memory of a thread-block cluster (rows spread over its CTAs);
//   k_bisect  : every eigenvalue of T by bisection on the Sturm sequence count (Barth, Martin &
//               Wilkinson), one thread per eigenvalue index, ascending by construction.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "am1gpu_internal.h"
#include "dmma_gemm.cuh"
#include "kernels.h"

namespace am1 {

namespace cg = cooperative_groups;

// Householder reduction of one symmetric matrix held on chip.  The n x n matrix is distributed by
// rows over a thread-block cluster of C CTAs (row r lives in CTA r % C, at local row r / C, full
// length n), so the whole reduction runs out of shared memory; C is the smallest cluster whose
// share fits one CTA.  Reflector s (GVL Alg. 8.3.1) zeroes row/column s below the subdiagonal:
// v_s = x + sign(x0)|x| e1 from x = A[s, s+1:], beta_s = 1/(|x|(|x| + |x0|)), and the trailing
// block takes the rank-2 update A -= v w^T + w v^T with p = beta A v, w = p - (beta/2)(p.v) v.
// Iteration s of the loop (update s-1 is on row s, reflector s is in row s's owner):
//   cluster barrier; the other CTAs copy v_s (distributed shared memory)
//   (b) one fused pass over the CTA's rows > s, a thread per pair of columns and group of rows: apply update
//       s-1 and accumulate this CTA's share of A v_s (A symmetric: column r of the share is a dot product
//       down the rows, so consecutive threads read consecutive words)
//   cluster barrier: every CTA's share ready; each CTA sums the C shares itself -> p, w_s, a thread per column
//   (a) the owner of row s+1 applies update s to it, the same threads on the same columns, and derives
//       reflector s+1
// Bound by shared memory traffic in (b) and by the latency of the four reductions and barriers elsewhere: with two
// columns to a thread and (v, w) in one word a row of 64 columns takes 10 wavefronts, against 14 with a column
// and three vectors; (a) by all threads follows (p.v) without a barrier of its own (a warp took 1440 cycles).
// One 192-row matrix (two CTAs, then one from 166 rows on) 768 -> 651 us, 192 molecules of 79 atoms 3.83 -> 3.29 ms.
// Column s below the diagonal is never read again: row s holds the same numbers and is the one read.
// All control flow is uniform over the cluster, so every CTA takes the same barriers.
// With job.stop > 0 the loop ends after reflector stop - 1: the trailing block (rows and columns
// >= stop) with update stop - 1 applied goes to job.W (row-major, n - stop rows), and a job on fewer
// CTAs reduces it as a matrix of its own, writing d and e from index stop on.  Its tridiagonal
// continues this one's: the block's reflectors act on indices >= stop + 1 and leave e[stop - 1] as is.
constexpr int TRI_THREADS = 512;
constexpr int TRI_WARPS = TRI_THREADS / 32;

// Dynamic shared memory of one CTA: local rows (even length), (v, w) (two buffers), the share of A v, 1 / beta (two
// buffers), beta and p of the next reflector's first column, two reduction scratches and the row groups' column sums.
size_t tridiag_smem_bytes(int n, int C) {
    const size_t rows = (size_t)(n + C - 1) / C, ld = (size_t)n + (n & 1);
    return sizeof(double) * (rows * ld + 5 * ld + 4 + 2 * TRI_WARPS + TRI_THREADS);
}

// The sum of the warps' partial sums in a tree: 16 dependent additions would be 130 cycles of every step, twice.
__device__ __forceinline__ double tri_warp_sums(const double* red) {
    double t[TRI_WARPS];
#pragma unroll
    for (int q = 0; q < TRI_WARPS; ++q) t[q] = red[q];
#pragma unroll
    for (int h = TRI_WARPS / 2; h > 0; h >>= 1)
#pragma unroll
        for (int q = 0; q < h; ++q) t[q] += t[q + h];
    return t[0];
}

__global__ void __launch_bounds__(TRI_THREADS) k_tridiag(const TriJob* __restrict__ jobs, const int* __restrict__ skip) {
    cg::cluster_group cluster = cg::this_cluster();
    const int C = (int)cluster.num_blocks();
    const int crank = (int)cluster.block_rank();
    const TriJob jb = jobs[blockIdx.x / C];
    if (skip && *skip) return;  // uniform over the cluster
    const int n = jb.n;
    const int ld = n + (n & 1);
    const int R = (n + C - 1) / C;
    extern __shared__ double2 tri_sh[];
    double* A = (double*)tri_sh;                      // R x ld: global row lr * C + crank at local row lr
    double2* vwb = (double2*)(A + (size_t)R * ld);    // (v, w), two buffers of ld (global column index)
    double* pp = (double*)(vwb + 2 * (size_t)ld);     // this CTA's share of A v
    double* bb = pp + ld;                             // 1 / beta, two buffers
    double* p1 = bb + 2;                              // beta_s, p of column s + 1
    double* red = p1 + 2;                             // [TRI_WARPS] p.v
    double* redn = red + TRI_WARPS;                   // [TRI_WARPS] |x|^2
    double* red2 = redn + TRI_WARPS;                  // [TRI_THREADS] column sums of the row groups
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto csync = [&]() {
        if (C > 1) cluster.sync();
        else __syncthreads();
    };
    // Row s (in its owner): the update with (v, w) = vw, whose entries of column s are vs, ws, and the reflector s
    // of the result into vn, d[s], e[s], with 1 / beta in *rb (0: no reflection).  A thread per column, s + tid; ends
    // with thread 1's vn[s + 1] and *rb not yet visible.
    auto reflect = [&](int s, const double2* vw, double vs, double ws, double2* vn, double* rb) {
        double* row = A + (size_t)(s / C) * ld;
        const bool has_next = s + 2 < n;
        double nrm = 0.0;
        for (int c = s + tid; c < n; c += TRI_THREADS) {
            const double2 q = vw[c];
            const double y = row[c] - vs * q.y - ws * q.x;
            row[c] = y;
            if (c > s) {
                vn[c].x = y;
                nrm = fma(y, y, nrm);
            }
        }
        if (!has_next) return;  // uniform over the CTA
        for (int o = 16; o > 0; o >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
        if (lane == 0) redn[warp] = nrm;
        __syncthreads();
        if (tid == 0) jb.d[s] = row[s];
        if (tid == 1) {
            const double alpha = sqrt(tri_warp_sums(redn)), x0 = row[s + 1];
            const double sg = x0 >= 0.0 ? 1.0 : -1.0;
            if (alpha != 0.0) vn[s + 1].x = x0 + sg * alpha;
            *rb = alpha * (alpha + fabs(x0));
            jb.e[s] = alpha == 0.0 ? 0.0 : -sg * alpha;
        }
    };
    for (int lr = warp; lr < R; lr += TRI_WARPS) {
        const int r = lr * C + crank;
        if (r >= n) break;
        for (int c = lane; c < ld; c += 32) A[(size_t)lr * ld + c] = c < n ? jb.A[(size_t)r * n + c] : 0.0;
    }
    for (int c = tid; c < 2 * ld; c += TRI_THREADS) vwb[c] = double2{0.0, 0.0};  // update "-1" is the identity
    __syncthreads();
    if (crank == 0) reflect(0, vwb + ld, 0.0, 0.0, vwb, bb);
    for (int s = 0; s + 1 < n; ++s) {
        const int nxt = s & 1;
        const double2* vw = vwb + (size_t)(1 - nxt) * ld;  // v, w of step s - 1
        double2* vn = vwb + (size_t)nxt * ld;              // of step s
        const bool has_next = s + 2 < n;
        const int owner = s % C;
        // (b) columns > s in pairs from an even one on (column s among them for an even s: written, not read), rows
        // c > s of this CTA.  Threads in G groups of a thread per pair; group g takes rows lr0 + g, lr0 + g + G, ...
        // (more groups when there are few columns, as many as red2 holds the sums of)
        const int lr0 = (s + 1 - crank + C - 1) / C;  // first local row with global index > s
        const int lre = (n - crank + C - 1) / C;      // local rows with global index < n
        const int q0 = (s + 1) & ~1;
        const int ncp = (n - q0 + 1) / 2;
        const int G = max(1, min(16, TRI_THREADS / (2 * ncp)));
        const int g = tid / ncp;
        csync();  // v_s ready in the owner, w_{s-1} everywhere
        if (has_next && crank != owner) {
            const double2* rv = cluster.map_shared_rank(vn, owner);
            for (int c = s + 1 + tid; c < n; c += TRI_THREADS) vn[c].x = rv[c].x;
            if (tid == 0) bb[nxt] = *cluster.map_shared_rank(bb + nxt, owner);
            __syncthreads();
        }
        if (tid == TRI_THREADS - 1 && has_next) *p1 = bb[nxt] == 0.0 ? 0.0 : 1.0 / bb[nxt];  // a thread (b) has no pair for
        for (int j = G > 1 ? tid - g * ncp : tid; j < ncp && (G == 1 || g < G); j += TRI_THREADS) {
            const int r = q0 + 2 * j;
            const double2 q = vw[r], q1 = vw[r + 1];
            double acc0 = 0.0, acc1 = 0.0;
            auto row2 = [&](double2 x, double2 m) {  // m: (v, w) of the row
                x.x = x.x - m.x * q.y - m.y * q.x;
                x.y = x.y - m.x * q1.y - m.y * q1.x;
                return x;
            };
            int lr = lr0 + (G > 1 ? g : 0);
            double2* ap = (double2*)(A + (size_t)lr * ld + r);
            const size_t step = (size_t)G * ld / 2;
            for (; lr + 3 * G < lre; lr += 4 * G, ap += 4 * step) {  // four independent rows per trip
                const int c0 = lr * C + crank, c1 = c0 + G * C, c2 = c1 + G * C, c3 = c2 + G * C;
                const double2 x0 = ap[0], x1 = ap[step], x2 = ap[2 * step], x3 = ap[3 * step];
                const double2 m0 = vw[c0], m1 = vw[c1], m2 = vw[c2], m3 = vw[c3];
                const double n0 = vn[c0].x, n1 = vn[c1].x, n2 = vn[c2].x, n3 = vn[c3].x;
                const double2 y0 = row2(x0, m0), y1 = row2(x1, m1), y2 = row2(x2, m2), y3 = row2(x3, m3);
                ap[0] = y0;
                ap[step] = y1;
                ap[2 * step] = y2;
                ap[3 * step] = y3;
                acc0 = fma(y0.x, n0, acc0), acc1 = fma(y0.y, n0, acc1);
                acc0 = fma(y1.x, n1, acc0), acc1 = fma(y1.y, n1, acc1);
                acc0 = fma(y2.x, n2, acc0), acc1 = fma(y2.y, n2, acc1);
                acc0 = fma(y3.x, n3, acc0), acc1 = fma(y3.y, n3, acc1);
            }
            if (lr < lre) {  // up to three more, their loads together
                const int k1 = lr + G < lre ? 1 : 0, k2 = lr + 2 * G < lre ? 2 : 0;
                const int c0 = lr * C + crank, c1 = c0 + k1 * G * C, c2 = c0 + k2 * G * C;
                const double2 x0 = ap[0], x1 = ap[k1 * step], x2 = ap[k2 * step];
                const double2 m0 = vw[c0], m1 = vw[c1], m2 = vw[c2];
                const double n0 = vn[c0].x, n1 = vn[c1].x, n2 = vn[c2].x;
                const double2 y0 = row2(x0, m0), y1 = row2(x1, m1), y2 = row2(x2, m2);
                ap[0] = y0;
                acc0 = fma(y0.x, n0, acc0), acc1 = fma(y0.y, n0, acc1);
                if (k1) {
                    ap[step] = y1;
                    acc0 = fma(y1.x, n1, acc0), acc1 = fma(y1.y, n1, acc1);
                }
                if (k2) {
                    ap[2 * step] = y2;
                    acc0 = fma(y2.x, n2, acc0), acc1 = fma(y2.y, n2, acc1);
                }
            }
            double* o = G > 1 ? red2 + 2 * (g * ncp + j) : pp + r;
            o[0] = acc0;
            o[1] = acc1;
            if (G > 1) break;
        }
        if (!has_next) break;
        if (G > 1) {
            __syncthreads();
            for (int r = s + 1 + tid; r < n; r += TRI_THREADS) {  // the loop below: the same thread's columns
                const double* col = red2 + r - q0;
                double t[4] = {0.0, 0.0, 0.0, 0.0};
                for (int q = 0; q < G; q += 4)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (q + k < G) t[k] += col[2 * (q + k) * ncp];
                pp[r] = (t[0] + t[1]) + (t[2] + t[3]);
            }
        }
        if (C > 1 || G == 1) csync();  // every CTA's share of A v_s ready
        const double beta = *p1;
        double part = 0.0;
        for (int r = s + 1 + tid; r < n; r += TRI_THREADS) {
            double sum = 0.0;
            if (C == 1) sum = pp[r];
            else
                for (int q = 0; q < C; ++q) sum += *cluster.map_shared_rank(pp + r, q);
            const double p = beta * sum;
            if (r == s + 1) p1[1] = p;
            vn[r].y = p;  // p for now, w below
            part = fma(p, vn[r].x, part);
        }
        for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        if (lane == 0) red[warp] = part;
        __syncthreads();
        const double kk = 0.5 * beta * tri_warp_sums(red);
        for (int r = s + 1 + tid; r < n; r += TRI_THREADS) vn[r].y = fma(-kk, vn[r].x, vn[r].y);
        if (s + 1 == jb.stop) {  // uniform over the cluster
            // hand-off: the trailing block with update s applied, to W (m x m, row-major)
            __syncthreads();
            const int s0 = s + 1, m = n - s0;
            for (int lr = (s0 - crank + C - 1) / C + warp; lr < R; lr += TRI_WARPS) {
                const int c = lr * C + crank;
                if (c >= n) break;
                const double2 m2 = vn[c];
                const double* arow = A + (size_t)lr * ld;
                double* out = jb.W + (size_t)(c - s0) * m - s0;
                for (int r = s0 + lane; r < n; r += 32) out[r] = arow[r] - m2.x * vn[r].y - m2.y * vn[r].x;
            }
            csync();  // no CTA leaves while another may still address its shared memory
            return;
        }
        // (a) row s + 1: its columns are those of w this thread wrote
        if (crank == (s + 1) % C) {
            const double v1 = vn[s + 1].x;
            reflect(s + 1, vn, v1, fma(-kk, v1, p1[1]), vwb + (size_t)(1 - nxt) * ld, bb + (1 - nxt));
        }
    }
    __syncthreads();
    // the last 2 x 2 block (or the 1 x 1 matrix)
    if (tid == 0) {
        if (n >= 2) {
            if ((n - 2) % C == crank) {
                jb.d[n - 2] = A[(size_t)((n - 2) / C) * ld + n - 2];
                jb.e[n - 2] = A[(size_t)((n - 2) / C) * ld + n - 1];
            }
            if ((n - 1) % C == crank) jb.d[n - 1] = A[(size_t)((n - 1) / C) * ld + n - 1];
        } else if (crank == 0) {
            jb.d[0] = A[0];
        }
    }
    csync();  // no CTA leaves while another may still address its shared memory
}

// Householder reduction of one matrix too large for a cluster's shared memory (n > ~448), by a
// group of G CTAs: the whole GPU (one cooperative launch per matrix) or a thread-block cluster
// (one cluster per matrix, all such matrices of a batch in one launch).  The matrix is copied to
// W (global memory, row-major), row r belongs to CTA r % G, and every step takes two group
// barriers.  Step s, as in k_tridiag:
//   every CTA stages v_{s-1} and w_{s-1} = p_{s-1} - kk_{s-1} v_{s-1} (columns >= s) in shared
//   memory
//   (a) the CTA owning row s applies update s-1 to it (all its threads, a column each) and derives
//       reflector s (a block reduction for the norm): v_s into global scratch, beta_s, d[s], e[s]
//   group barrier; every CTA stages v_s
//   (b) every CTA, a warp per own row r > s: apply update s-1 to row r (columns > s) and form
//       p_r = beta_s W[r, s+1:] . v_s in the same pass; the CTA's share of p.v.  Bound by the latency
//       of those loads: each lane loads TRIB_BATCH elements of two rows before it stores any
//       (nine matrices of more than 630 rows, 16 CTAs each, 19.4 -> 15.7 ms against one row).
//   group barrier
//   every warp sums the G shares in the same order, so all hold the same kk_s = beta_s (p.v) / 2.
// Global scratch (job.work): v[2][n] | p[2][n] | share[G] | beta[2]; dynamic shared memory: 3 n
// doubles (tridiag_big_smem_bytes).  Row s of W ends holding reflector v_s in columns s+1..n-1
// (its first entry corrected after the norm), for the eigenvector back-transformation.
constexpr int TRIB_BATCH = 8;

size_t tridiag_big_smem_bytes(int n) { return sizeof(double) * 3 * (size_t)n; }

template <class Sync>
__device__ void tridiag_group(const TriJob& jb, int G, int gi, Sync sync) {
    const int n = jb.n;
    double* W = jb.W;
    double* vb = jb.work;              // v_s, two buffers
    double* pb = vb + 2 * (size_t)n;   // p_s, two buffers
    double* share = pb + 2 * (size_t)n;
    double* bb = share + G;            // beta_s, two buffers
    extern __shared__ double tsh[];
    double* sv = tsh;           // v_{s-1}
    double* sw = tsh + n;       // w_{s-1}
    double* svn = tsh + 2 * n;  // v_s
    constexpr int NW = TRIB_THREADS / 32;
    __shared__ double red[NW];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto bsum = [&](double v) {
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        __syncthreads();
        if (lane == 0) red[warp] = v;
        __syncthreads();
        double t = 0.0;
        for (int q = 0; q < NW; ++q) t += red[q];
        return t;
    };
    // own rows into W; update "-1" is the identity: v = p = 0, kk = 0
    for (int r = gi + warp * G; r < n; r += NW * G)
        for (int c = lane; c < n; c += 32) W[(size_t)r * n + c] = jb.A[(size_t)r * n + c];
    for (int c = gi * TRIB_THREADS + tid; c < n; c += G * TRIB_THREADS) {
        vb[n + c] = 0.0;
        pb[n + c] = 0.0;
    }
    double kk = 0.0;
    sync();
    for (int s = 0; s + 1 < n; ++s) {
        const int cur = (s + 1) & 1, nxt = s & 1;
        const double* v = vb + (size_t)cur * n;  // reflector s - 1
        const double* p = pb + (size_t)cur * n;
        double* vn = vb + (size_t)nxt * n;       // reflector s
        double* pn = pb + (size_t)nxt * n;
        const bool has_next = s + 2 < n;
        for (int c = s + tid; c < n; c += TRIB_THREADS) {
            const double vc = __ldcg(v + c);
            sv[c] = vc;
            sw[c] = __ldcg(p + c) - kk * vc;
        }
        __syncthreads();
        if (gi == s % G) {  // (a)
            double* row = W + (size_t)s * n;
            const double vs = sv[s], ws = sw[s];
            double nrm = 0.0;
            for (int c = s + tid; c < n; c += TRIB_THREADS) {
                const double vc = sv[c];
                const double y = row[c] - vs * sw[c] - ws * vc;
                row[c] = y;
                if (c > s) {
                    vn[c] = y;
                    nrm += y * y;
                }
            }
            nrm = bsum(nrm);  // its barriers also make row[s], row[s + 1] visible to thread 0
            if (tid == 0) {
                const double alpha = sqrt(nrm), x0 = row[s + 1];
                const double sg = x0 >= 0.0 ? 1.0 : -1.0;
                jb.d[s] = row[s];
                if (has_next) {
                    jb.e[s] = alpha == 0.0 ? 0.0 : -sg * alpha;
                    bb[nxt] = alpha == 0.0 ? 0.0 : 1.0 / (alpha * (alpha + fabs(x0)));
                    if (alpha != 0.0) {
                        vn[s + 1] = x0 + sg * alpha;
                        row[s + 1] = x0 + sg * alpha;  // row s now holds v_s exactly (read by no later step)
                    }
                } else {
                    jb.e[s] = row[s + 1];  // the last 2 x 2 block: e[n-2]
                }
            }
        }
        sync();  // v_s and beta_s ready
        for (int c = s + 1 + tid; c < n; c += TRIB_THREADS) svn[c] = __ldcg(vn + c);
        __syncthreads();
        // (b) own rows r > s, a warp per row
        const double beta = has_next ? __ldcg(bb + nxt) : 0.0;
        double part = 0.0;
        const int r0 = s + 1 + ((gi - (s + 1) % G) % G + G) % G;  // first own row > s
        for (int r = r0 + warp * G; r < n; r += 2 * NW * G) {
            const int rb = r + NW * G;
            const bool two = rb < n;  // uniform over the warp
            double* rowa = W + (size_t)r * n;
            double* rowb = W + (size_t)(two ? rb : r) * n;
            const double va = sv[r], wa = sw[r], vb2 = two ? sv[rb] : 0.0, wb2 = two ? sw[rb] : 0.0;
            double acca = 0.0, accb = 0.0;
            for (int c0 = s + 1 + lane; c0 < n; c0 += 32 * TRIB_BATCH) {
                double x[TRIB_BATCH], z[TRIB_BATCH];
#pragma unroll
                for (int u = 0; u < TRIB_BATCH; ++u) {
                    const int c = c0 + 32 * u;
                    x[u] = c < n ? rowa[c] : 0.0;
                    z[u] = two && c < n ? rowb[c] : 0.0;
                }
#pragma unroll
                for (int u = 0; u < TRIB_BATCH; ++u) {
                    const int c = c0 + 32 * u;
                    if (c < n) {
                        const double vc = sv[c], wc = sw[c], nc = svn[c];
                        const double y = x[u] - va * wc - wa * vc;
                        rowa[c] = y;
                        acca = fma(y, nc, acca);
                        if (two) {
                            const double t = z[u] - vb2 * wc - wb2 * vc;
                            rowb[c] = t;
                            accb = fma(t, nc, accb);
                        }
                    }
                }
            }
            for (int o = 16; o > 0; o >>= 1) {
                acca += __shfl_xor_sync(0xffffffffu, acca, o);
                accb += __shfl_xor_sync(0xffffffffu, accb, o);
            }
            const double pa = beta * acca, pb2 = beta * accb;
            if (lane == 0 && has_next) {
                pn[r] = pa;
                if (two) pn[rb] = pb2;
            }
            part += pa * svn[r];
            if (two) part += pb2 * svn[rb];
        }
        if (!has_next) break;
        part = bsum(lane == 0 ? part : 0.0);
        if (tid == 0) share[gi] = part;
        sync();  // p_s and every share ready
        kk = 0.5 * beta * group_share_sum(share, G);
    }
    __syncthreads();
    if (n == 1 && gi == 0 && tid == 0) jb.d[0] = W[0];
    if (n >= 2 && gi == (n - 1) % G && tid == 0) jb.d[n - 1] = W[(size_t)(n - 1) * n + n - 1];
}

__global__ void __launch_bounds__(TRIB_THREADS) k_tridiag_big(TriJob jb) {
    cg::grid_group grid = cg::this_grid();
    tridiag_group(jb, (int)gridDim.x, (int)blockIdx.x, [&] { grid.sync(); });
}

// One cluster (gridDim.x CTAs) per matrix of jobs[blockIdx.y].
__global__ void __launch_bounds__(TRIB_THREADS) k_tridiag_cl(const TriJob* __restrict__ jobs) {
    cg::cluster_group cl = cg::this_cluster();
    tridiag_group(jobs[blockIdx.y], (int)cl.num_blocks(), (int)cl.block_rank(), [&] { cl.sync(); });
}

// Number of eigenvalues of T below x: the sign changes of the leading principal minors
// p_i = (d_i - x) p_{i-1} - e_{i-1}^2 p_{i-2} (p_{-1} = 1), the Sturm sequence of the
// tridiagonal.  Same count as the LDL^T pivots q_i = p_i / p_{i-1} < 0, without the division on the
// critical path (one FMA per step).  The pair (p_{i-1}, p_{i-2}) is rescaled by a power of two
// every 8 steps (exact), which keeps it far from overflow and underflow; a zero p_i is replaced by a
// tiny multiple of p_{i-1} (a zero pivot counts as non-negative, as in the division form).
// Eight steps go without a test on the critical path (one FMA a step; signs and zeros are read off the high
// words beside it); a block that met a zero is taken again with the replacement.
__device__ __forceinline__ int sturm_count(const double2* de, int n, double x) {
    double p2 = 1.0;
    double p1 = de[0].x - x;
    if (p1 == 0.0) p1 = 0x1p-200;
    int sign = __double2hiint(p1);  // of p1, in the top bit
    int c = (unsigned)sign >> 31;
    for (int i = 1; i < n; i += 8) {
        const int m = min(8, n - i);
        bool zero = m < 8;
        if (!zero) {
            double q2 = p2, q1 = p1;
            int s = sign, cc = 0;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const double2 r = de[i + u];
                const double p = fma(r.x - x, q1, -r.y * q2);
                const int h = __double2hiint(p);
                zero |= ((h << 1) | __double2loint(p)) == 0;
                cc += (unsigned)(h ^ s) >> 31;
                s = h;
                q2 = q1;
                q1 = p;
            }
            if (!zero) {
                p2 = q2;
                p1 = q1;
                sign = s;
                c += cc;
            }
        }
        if (zero) {
            for (int u = 0; u < m; ++u) {
                const double2 r = de[i + u];
                double p = fma(r.x - x, p1, -r.y * p2);
                if (p == 0.0) p = 0x1p-200 * p1;
                const int h = __double2hiint(p);
                c += (unsigned)(h ^ sign) >> 31;
                sign = h;
                p2 = p1;
                p1 = p;
            }
        }
        const int ex = max(__double2hiint(p1) & 0x7fffffff, __double2hiint(p2) & 0x7fffffff) >> 20;  // biased, of the larger
        if (ex > 1423 || ex < 623) {
            const double sc = __longlong_as_double((long long)(2046 - ex) << 52);  // 2^-(ex - 1023)
            p1 *= sc;
            p2 *= sc;
        }
    }
    return c;
}

// Eigenvalue k of T by bisection to the width 4 eps max(|lo|, |hi|).  lanes = 1: a thread per eigenvalue;
// lanes = 32: a warp per eigenvalue, five levels of the bisection per round, the 31 midpoints that five steps can
// reach counted on the lanes and the steps then walked; for launches with few eigenvalues, where the latency
// of one thread's ~50 dependent counts is the cost.  The midpoints, the counts and so
// the eigenvalues are the same either way.  n = 1501: 5.0 -> 0.7 ms, 192 orbitals alone 107 -> 83 us (32-way multisection
// before, whose eigenvalues differed from the thread form's in the last bits), a batch of 192 molecules 1.07 -> 0.83 ms.
__global__ void k_bisect(const TriJob* __restrict__ jobs, const int* __restrict__ skip, int lanes) {
    const TriJob jb = jobs[blockIdx.x];
    if (skip && *skip) return;
    const int n = jb.n;
    extern __shared__ __align__(16) double sh[];
    double2* de = reinterpret_cast<double2*>(sh);  // d_i, e_{i-1}^2
    __shared__ double bounds[2], wlo[32], whi[32];
    double lo_t = 1e300, hi_t = -1e300;  // Gershgorin bounds of T (every thread's share, then the CTA's)
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const double di = jb.d[i], er = i + 1 < n ? jb.e[i] : 0.0, el = i > 0 ? jb.e[i - 1] : 0.0;
        de[i] = make_double2(di, el * el);
        const double r = fabs(el) + fabs(er);
        lo_t = fmin(lo_t, di - r);
        hi_t = fmax(hi_t, di + r);
    }
    for (int o = 16; o > 0; o >>= 1) {
        lo_t = fmin(lo_t, __shfl_xor_sync(0xffffffffu, lo_t, o));
        hi_t = fmax(hi_t, __shfl_xor_sync(0xffffffffu, hi_t, o));
    }
    if ((threadIdx.x & 31) == 0) {
        wlo[threadIdx.x >> 5] = lo_t;
        whi[threadIdx.x >> 5] = hi_t;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double lo = 1e300, hi = -1e300;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            lo = fmin(lo, wlo[w]);
            hi = fmax(hi, whi[w]);
        }
        const double pad = 1e-12 * fmax(fabs(lo), fabs(hi)) + 1e-300;
        bounds[0] = lo - pad;
        bounds[1] = hi + pad;
    }
    __syncthreads();
    if (lanes == 32) {
        const int k = (blockIdx.y * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
        if (k >= n) return;  // whole warps: blockDim is a multiple of 32
        double lo = bounds[0], hi = bounds[1];
        bool done = false;
        for (int round = 0; round < 40 && !done; ++round) {
            // lane's node of the tree, in heap order (node 0 the root, children 2 i + 1 below and 2 i + 2
            // above its midpoint): the interval that its parents' answers would leave
            double l = lo, h = hi, mid = 0.5 * (lo + hi);
            const int node = lane + 1;  // 1-based; lane 31 idles
            for (int bit = 30 - __clz(node); bit >= 0; --bit) {
                if (node >> bit & 1) l = mid;
                else h = mid;
                mid = 0.5 * (l + h);
            }
            const bool halt = !(mid > l && mid < h) || h - l <= 4.0 * 2.220446049250313e-16 * fmax(fabs(l), fabs(h));
            const bool up = lane < 31 && !halt && sturm_count(de, n, mid) <= k;
            const unsigned halts = __ballot_sync(0xffffffffu, halt), ups = __ballot_sync(0xffffffffu, up);
            // the steps, on the nodes' bits alone (each step's own arithmetic cost a matrix of 5 rows 5 of 45 us): to the
            // node where bisection ends, or past the last of five
            int at = 1, last = 1;
            for (int step = 0; step < 5 && !done; ++step) {
                done = halts >> (at - 1) & 1;
                last = at;
                at = 2 * at + (ups >> (at - 1) & 1);
            }
            lo = __shfl_sync(0xffffffffu, !done && up ? mid : l, last - 1);
            hi = __shfl_sync(0xffffffffu, done || up ? h : mid, last - 1);
        }
        if (lane == 0) jb.eps[k] = 0.5 * (lo + hi);
        return;
    }
    const int k0 = blockIdx.y * blockDim.x;  // this block's share of the eigenvalue indices
    if (k0 >= n) return;
    for (int k = k0 + threadIdx.x; k < min(n, k0 + (int)blockDim.x); k += blockDim.x) {
        double lo = bounds[0], hi = bounds[1];
        for (int it = 0; it < 200; ++it) {
            const double mid = 0.5 * (lo + hi);
            if (!(mid > lo && mid < hi)) break;
            if (hi - lo <= 4.0 * 2.220446049250313e-16 * fmax(fabs(lo), fabs(hi))) break;
            if (sturm_count(de, n, mid) <= k) lo = mid;
            else hi = mid;
        }
        jb.eps[k] = 0.5 * (lo + hi);
    }
}

}  // namespace am1

namespace am1 {

// ---------------------------------------------------------------------------------------------
// Blocked Householder reduction for the largest matrices (the whole GPU per matrix): panels of
// TRP_B columns, each reduced by one cooperative launch (k_tridiag_panel, the DLATRD scheme) with
// the trailing matrix left untouched, then the trailing matrix updated once per panel,
// A <- A - V W^T - W V^T, by a rank-2 TRP_B product on the FP64 tensor cores (k_tridiag_syr2k*).
// Per column the panel kernel reads the trailing matrix once (A v) instead of reading and writing
// it (the unblocked k_tridiag_big), and the writes happen once per panel.
//
// Column c = k + j of the panel (V, W: the panel's reflectors and their w vectors so far, rows
// > c; V_c., W_c. row c of them):
//   x_i  = A_ic - sum_{l<j} (V_il W_cl + W_il V_cl)               i >= c   (column c, updated)
//   d_c  = x_c;  alpha = |x_{c+1:}|,  v = x_{c+1:} + sign(x_{c+1}) alpha e_1,
//   beta = 1 / (alpha (alpha + |x_{c+1}|)),  e_c = -sign(x_{c+1}) alpha
//   p    = beta (A v - V (W^T v) - W (V^T v))                      over rows and columns > c
//   w    = p - (beta/2)(p . v) v,  V_.j = v,  W_.j = w
// W^T v and V^T v come from W^T x and V^T x (summed with |x|^2 in the first grid barrier) and
// row c+1 of W and V; they are needed only after the second barrier, which sums v . A v, since
// p . v = beta (v . A v - 2 (V^T v) . (W^T v)).  Two grid barriers per column: row c+1's newest
// entries of V and W, which its owner writes after the second barrier, every CTA forms itself for
// the next column's first phase.  Rows are cyclic over G shares (r % G), the CTAs of a GPU that the matrix has to
// itself; fewer CTAs take several shares each, with the same sums in the same order, so the results do not depend on
// how many there are (blocked_tridiag).
// Scratch (job.work, 16-byte aligned): VW[n][2B] = [V | W] | WVt[2B][n] = [W | V]^T | x[n] |
// u[n] | share[2B + 2][G] | sums[2B]; dynamic shared memory: v (n doubles) and W^T v, V^T v.  As in
// tridiag_group, row c of job.W ends holding reflector v_c in columns c+1..n-1.
// ---------------------------------------------------------------------------------------------

size_t tridiag_panel_smem_bytes(int n) { return sizeof(double) * ((size_t)n + 2 * TRP_B); }

// Sum over the CTAs of one slot's shares (consecutive words) by a warp: lane-strided in ascending order, then
// a butterfly, as group_share_sum; up to 160 shares' loads are in flight at once.
__device__ __forceinline__ double panel_share_sum(const double* __restrict__ share, int G) {
    constexpr int U = 5;
    const int lane = threadIdx.x & 31;
    double t = 0.0;
    for (int q0 = 0; q0 < G; q0 += 32 * U) {
        double v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = q0 + 32 * u + lane < G ? __ldcg(share + q0 + 32 * u + lane) : 0.0;
#pragma unroll
        for (int u = 0; u < U; ++u) t += v[u];
    }
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
}

// Bound by the chain of a column: two grid barriers (2.5k cycles each), the L2 round trips between them, and
// from about 1500 rows on the pass over the trailing matrix.  In its first form every CTA summed every slot's
// shares itself, from records a CTA apart: 60 MB of L2 sectors per column (clock stamps at n = 1501, cycles per
// column: 4.1k for the column, 15.7k for the reflector, 6.7k for A v, 8.7k for w).  Now a slot is summed by one CTA,
// from consecutive words, while the others multiply, and A v's rows are reduced behind one barrier: 2.5k, 3.2k, 8.2k and
// 2.3k; eigenvalues alone, with copies and bisection, 1501 rows 34.8 -> 17.5 ms, 3072 rows 92 -> 53 ms.
__global__ void __launch_bounds__(TRIB_THREADS) k_tridiag_panel(TriJob jb, int k, int bw, int G) {
    cg::grid_group grid = cg::this_grid();
    const int n = jb.n;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // the G shares of the work: CTA b takes b, b + gridDim.x, ..., L in all, 64 threads each for the work on single rows, S
    // rows' room each
    const int P = (int)gridDim.x, L = (G + P - 1) / P, S = 64 / L;
    const int lg = tid >> 6, t = tid & 63, gi = (int)blockIdx.x + lg * P;
    const bool act = lg < L && gi < G;
    constexpr int NW = TRIB_THREADS / 32;
    constexpr int B = TRP_B;
    double* A = jb.W;
    double* VW = jb.work;
    double* WVt = VW + (size_t)2 * B * n;
    double* xb = WVt + (size_t)2 * B * n;
    double* ub = xb + n;
    double* share = ub + n;                        // [2B + 2][G]: |x|^2, W^T x, V^T x (as the column has them), v.u
    double* sums = share + (size_t)(2 * B + 2) * G;  // [2B]: W^T v, V^T v
    extern __shared__ double psh[];
    double* sv = psh;      // v, rows c+1..n-1
    double* st = psh + n;  // [0, B): W^T v;  [B, 2B): V^T v
    __shared__ double xr[64];  // this CTA's x_i of the current column (its rows >= c, at most 64 of them)
    __shared__ double red[NW];
    // the panel's V and W on this CTA's own rows (row gi + q G of a share in its slot q), kept here as they are
    // formed: the per-column corrections read them from shared memory, not global
    __shared__ double svw[64][2 * TRP_B];
    __shared__ double srow[2 * TRP_B];  // V and W of row c (formed locally in the previous column, or read)
    __shared__ double redr[64][NW];     // A v of the own rows, each warp's part of the columns
    // rows >= c = cd G + cm of share g: the first, how many (<= S), the slot of the first, the index of the first > c
    struct Rows {
        int first, nr, q0, qa;
    };
    const int nd = n / G, nm = n % G;
    int cd = k / G, cm = k % G;
    auto rows = [&](int g) {
        Rows r;
        r.q0 = cd + (g < cm ? 1 : 0);
        r.first = r.q0 * G + g;
        r.nr = nd + (g < nm ? 1 : 0) - r.q0;
        r.qa = g == cm ? 1 : 0;
        return r;
    };
    for (int j = 0; j < bw; ++j) {
        const int c = k + j;
        if (j > 0 && ++cm == G) {
            cm = 0;
            ++cd;
        }
        __syncthreads();  // own rows' V, W of the previous column, and srow, are written
        // ---- phase 1: column c for own rows i >= c, and this CTA's shares of |x|^2, W^T x, V^T x
        const Rows me = rows(gi);
        const int row = me.first + t * G, slot0 = lg * S + me.q0, at = lg * S;  // this thread's own row (where t < nr)
        if (act && t < me.nr) {
            const int i = row;
            const double* Vi = svw[slot0 + t];
            double x = __ldcg(A + (size_t)i * n + c);
            for (int l = 0; l < j; ++l) x -= Vi[l] * srow[B + l] + Vi[B + l] * srow[l];
            xr[at + t] = x;
            xb[i] = x;
            if (i == c) jb.d[c] = x;
        }
        __syncthreads();
        if (act && t < 2 * j + 1) {  // share slot 0: |x_{>c}|^2; 1..j: W^T x; j+1..2j: V^T x
            double s = 0.0;
            for (int q = me.qa; q < me.nr; ++q) {
                const double xq = xr[at + q];
                if (t == 0) s += xq * xq;
                else if (t <= j) s += svw[slot0 + q][B + (t - 1)] * xq;
                else s += svw[slot0 + q][t - 1 - j] * xq;
            }
            share[(size_t)t * G + gi] = s;
        }
        grid.sync();
        // ---- the reflector (every CTA forms the same values: fixed-order sums of the shares)
        const bool has_next = c + 2 < n;
        const double x1 = __ldcg(xb + c + 1);
        if (!has_next) {  // the last 2 x 2 block: e[n-2], and d[n-1] with this panel's updates
            if (act && gi == (nm == 0 ? G - 1 : nm - 1) && t == 0) {
                jb.e[c] = x1;
                double dn = __ldcg(A + (size_t)(n - 1) * n + n - 1);
                const double* Vn = VW + (size_t)(n - 1) * 2 * B;
                for (int l = 0; l < j; ++l) dn -= 2.0 * __ldcg(Vn + l) * __ldcg(Vn + B + l);
                jb.d[n - 1] = dn;
            }
            break;
        }
        for (int i0 = c + 1 + tid; i0 < n; i0 += 4 * TRIB_THREADS) {
            double v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = i0 + u * TRIB_THREADS < n ? __ldcg(xb + i0 + u * TRIB_THREADS) : 0.0;
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (i0 + u * TRIB_THREADS < n) sv[i0 + u * TRIB_THREADS] = v[u];
        }
        // |x|^2 in warp 0; the slots (W^T x or V^T x) of the shares one each in the CTAs' warps 1, then 2, and so on,
        // summed for all CTAs: warp 1 alone where there are 2 B CTAs
        const double* V1 = VW + (size_t)(c + 1) * 2 * B;
        const int sl = (int)blockIdx.x + (warp - 1) * P;
        const bool slot = warp > 0 && sl < 2 * j;
        const double sum = warp == 0 ? panel_share_sum(share, G) : slot ? panel_share_sum(share + (size_t)(1 + sl) * G, G) : 0.0;
        const double v1 = slot ? __ldcg(V1 + (sl < j ? B + sl : sl - j)) : 0.0;
        if (warp == 0 && lane == 0) red[0] = sum;
        __syncthreads();
        const double alpha = sqrt(red[0]);
        const double sg = x1 >= 0.0 ? 1.0 : -1.0;
        const double beta = alpha == 0.0 ? 0.0 : 1.0 / (alpha * (alpha + fabs(x1)));
        if (slot && lane == 0)  // plus the e_{c+1} part of v = x + sg alpha e_{c+1}
            sums[sl < j ? sl : B + sl - j] = sum + sg * alpha * v1;
        if (tid == 0) sv[c + 1] = x1 + sg * alpha;
        __syncthreads();
        // ---- phase 2a: u = A v on own rows i > c, this CTA's share of v . u.  Rows go in groups of
        // four; every thread takes a stride of the columns for all four (many loads in flight),
        // and the partial sums are reduced over the CTA in a fixed order.
        for (int l = 0, g = (int)blockIdx.x; l < L && g < G; ++l, g += P) {
            const Rows r = rows(g);
            for (int g0 = r.qa; g0 < r.nr; g0 += 4) {
                const int gr = min(4, r.nr - g0);
                const double* Ar[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) Ar[u] = A + (size_t)(r.first + (g0 + (u < gr ? u : 0)) * G) * n;
                double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 2
                for (int m = c + 1 + tid; m < n; m += TRIB_THREADS) {
                    const double vm = sv[m];
#pragma unroll
                    for (int u = 0; u < 4; ++u) acc[u] = fma(__ldcg(Ar[u] + m), vm, acc[u]);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    for (int o = 16; o > 0; o >>= 1) acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], o);
                if (lane == 0)
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (u < gr) redr[l * S + g0 + u][warp] = acc[u];
            }
        }
        __syncthreads();
        const bool own = act && t >= me.qa && t < me.nr;
        double ui = 0.0;  // u of this thread's own row, kept for phase 2b
        if (lg < L) {
            double part = 0.0;
            if (own) {
                for (int w = 0; w < NW; ++w) ui += redr[at + t][w];
                if (row == c + 1) ub[row] = ui;
                part = ui * sv[row];
            }
            for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
            if (lane == 0) red[1 + warp] = part;
        }
        __syncthreads();
        if (act && t == 0) share[(size_t)(2 * B + 1) * G + gi] = red[1 + 2 * lg] + red[2 + 2 * lg];
        grid.sync();
        // ---- phase 2b: p = beta (u - V (W^T v) - W (V^T v)), w = p - kk v for own rows i > c with
        // kk = (beta / 2) p . v, p . v = beta (v . u - 2 (V^T v) . (W^T v)); column j of V and W in both
        // layouts; and row c + 1 of V and W (its p formed by every CTA) for the next column's phase 1
        if (warp == 0) {
            const double vu = panel_share_sum(share + (size_t)(2 * B + 1) * G, G);
            if (lane == 0) red[0] = vu;
        } else if (warp < 1 + 2 * B / 32) {
            const int e = tid - 32, l = e < B ? e : e - B;
            if (l < j) st[e] = __ldcg(sums + e);
        } else if (warp < 1 + 4 * B / 32) {
            const int e = tid - 32 - 2 * B, l = e < B ? e : e - B;
            if (l < j) srow[e] = __ldcg(V1 + e);  // [V | W], as VW's rows
        }
        const double u1 = tid == TRIB_THREADS - 1 ? __ldcg(ub + c + 1) : 0.0;
        __syncthreads();
        const bool next_row = tid == TRIB_THREADS - 1;  // (no share's: L < 8)
        const double* Vi = next_row ? srow : svw[own ? slot0 + t : 0];
        double pu = next_row ? u1 : ui, vv = 0.0;
        if (own || next_row) {
            for (int l = 0; l < j; ++l) {
                pu -= Vi[l] * st[l] + Vi[B + l] * st[B + l];
                vv += st[l] * st[B + l];
            }
        }
        const double p = beta * pu, kk = 0.5 * beta * (beta * (red[0] - 2.0 * vv));
        if (own) {
            const int i = row;
            const double v = sv[i], w = p - kk * v;
            svw[slot0 + t][j] = v;
            svw[slot0 + t][B + j] = w;
            VW[(size_t)i * 2 * B + j] = v;
            VW[(size_t)i * 2 * B + B + j] = w;
            WVt[(size_t)j * n + i] = w;
            WVt[(size_t)(B + j) * n + i] = v;
            A[(size_t)c * n + i] = v;  // reflector c into row c (columns > c), which nothing reads again
        }
        if (next_row) {
            srow[j] = sv[c + 1];
            srow[B + j] = p - kk * sv[c + 1];
        }
        if (act && gi == cm && t == 0) jb.e[c] = alpha == 0.0 ? 0.0 : -sg * alpha;
    }
}

// A[t0 + r][t0 + q] -= (V W^T + W V^T)[t0 + r][t0 + q] over the upper-triangle 64 x 64 tiles of the
// trailing block (t0 = k + TRP_B), mirrored: C = [V | W][rows] . [W | V]^T[:, cols], K = 2 TRP_B.
template <bool PAIRS>
__device__ __forceinline__ void syr2k_body(TriJob jb, int t0) {
    extern __shared__ __align__(16) double dsm[];
    const int n = jb.n, T = n - t0;
    const int nt = (T + DG_TILE - 1) / DG_TILE;
    int rem = blockIdx.x, tm = 0;
    while (rem >= nt - tm) {
        rem -= nt - tm;
        ++tm;
    }
    const int tn = tm + rem;
    const int m0 = tm * DG_TILE, n0 = tn * DG_TILE;
    const double* VW = jb.work;
    const double* WVt = VW + (size_t)2 * TRP_B * n;
    const bool compute = dg_quarter_on(m0, n0, T, T, tm == tn);
    double acc[2][4][4];
    dg_mainloop<PAIRS>(dsm, VW + (size_t)t0 * 2 * TRP_B, 2 * TRP_B, WVt + t0, n, T, T, 2 * TRP_B, m0, n0, acc, compute);
    double* A = jb.W + (size_t)t0 * n + t0;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int r = m0 + dg_row(i, e), c = n0 + dg_col(j, e);
                if (compute && r <= c && c < T) {
                    const double y = A[(size_t)r * n + c] - acc[i][j][e];
                    A[(size_t)r * n + c] = y;
                    if (r < c) A[(size_t)c * n + r] = y;
                }
            }
}

__global__ void __launch_bounds__(DG_THREADS, 4) k_tridiag_syr2k16(TriJob jb, int t0) { syr2k_body<true>(jb, t0); }
__global__ void __launch_bounds__(DG_THREADS, 4) k_tridiag_syr2k8(TriJob jb, int t0) { syr2k_body<false>(jb, t0); }

}  // namespace am1
