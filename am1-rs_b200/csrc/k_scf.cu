// The per-iteration SCF bookkeeping kernels (am1-rs src/scf.rs:475-1204), batched over
// molecules and spin channels:
//   k_sad_init     superposition-of-atomic-densities guess            scf.rs:475-494, 730-740
//   k_commutator   the commutator e = FP - (FP)^T = F.P - P.F (scf.rs:531-544) straight from F and
//                  P on the FP64 tensor cores, upper-triangle tiles only; its epilogue pushes e
//                  into the packed history and forms |e|^2 (scf.rs:600) and the new row of the
//                  CDIIS Gram matrix, so F.P is never stored
//   k_post_fock    one pass over the upper triangle of F, P, H: energy traces (scf.rs:595, 767),
//                  the packed history push of F and P (scf.rs:603-614, 877-952) and the new
//                  row/column of the A-DIIS Gram matrix (only those change)
//   k_diis_solve   one thread per molecule: history bookkeeping, divergence guard
//                  (scf.rs:621-625), CDIIS bordered solve with the 1e-12 pivot guard
//                  (scf.rs:966-988, 1095-1141), A-DIIS simplex (scf.rs:1061-1091, 1144-1204)
//   k_combine      F* = sum c_i F_i from the packed history (scf.rs:955-963), Gershgorin bounds
//   k_density_post rms(P_new - P) and P <- P_new                      scf.rs:546-555
//   k_converge     de / dp test and iteration count                   scf.rs:663-696, 810-823
#include <cuda_runtime.h>

#include "am1gpu_internal.h"
#include "dmma_gemm.cuh"
#include "kernels.h"

namespace am1 {

__device__ __forceinline__ long long sym_row(int r, int n) { return (long long)r * n - (long long)r * (r - 1) / 2; }
__device__ __forceinline__ long long anti_row(int r, int n) { return (long long)r * n - (long long)r * (r + 1) / 2; }

__global__ void k_sad_init(const MolDesc* __restrict__ mols, const int* __restrict__ atom_mol, int natoms_total,
                           const DevElem* __restrict__ params, const int* __restrict__ atom_z, double* __restrict__ arena) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= natoms_total) return;
    const MolDesc md = mols[atom_mol[a]];
    const int A = a - md.atom_base, h = md.nheavy, n = md.nao;
    const DevElem& e = params[md.method * (MAX_Z + 1) + atom_z[a]];
    const double zv = e.core_charge;
    const double ns = fmin(zv, 2.0), np = fmax(zv - ns, 0.0);
    double scale[2] = {1.0, 1.0};
    if (md.nch == 2) {
        const double tot = (double)max(md.n_occ[0] + md.n_occ[1], 1);
        scale[0] = (double)md.n_occ[0] / tot;
        scale[1] = (double)md.n_occ[1] / tot;
    }
    for (int c = 0; c < md.nch; ++c) {
        double* P = arena + md.ch_base[c] + SLOT_P * (long long)n * n;
        if (A < h) {
            const int o = 4 * A;
            P[(long long)o * n + o] = ns * scale[c];
            for (int k = 1; k < 4; ++k) P[(long long)(o + k) * n + o + k] = np / 3.0 * scale[c];
        } else {
            const int o = 4 * h + (A - h);
            P[(long long)o * n + o] = ns * scale[c];
        }
    }
}

// Fresh SCF state for every molecule of a batch (each run starts from the SAD guess).
__global__ void k_state_init(MolState* __restrict__ st, const MolDesc* __restrict__ mols, int nmol, int lowp) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nmol) return;
    MolState s{};
    s.active = 1;
    // mixed precision: every closed shell, and the open shells that keep the eigensolver fallback
    // (at most kLowpMaxOpenShellAo orbitals).  Large radicals start FP64: a TF32 start left a few
    // of them (3 of about 1900 in a 100 000-request stream) in a UHF basin that CDIIS did not leave.
    s.lowp = lowp && (mols[i].nch == 1 || mols[i].nao <= kLowpMaxOpenShellAo);
    s.residual = __longlong_as_double(0x7ff0000000000000LL);  // +inf
    st[i] = s;
}

// F* = 0 (what the final spectrum is of where no iteration formed one: none allowed, or an energy that is not finite in the
// first), P = 0 (k_sad_init then sets its diagonal) and the eigensolver's warm start C^T = I: the three slots a run reads before
// it writes them.  Bound by the writes; the whole arena, six slots and more a channel, was zeroed for these, and twice in a
// batched call (25 GB each time for 4096 molecules, 7 ms a call).
__global__ void __launch_bounds__(256) k_slots_init(const ChanJob* __restrict__ jobs) {
    static_assert(SLOT_P == SLOT_FX + 1 && SLOT_CT == SLOT_P + 1, "F*, P and Ct adjacent");
    const ChanJob& jb = jobs[blockIdx.y];
    const int n = jb.n;
    double* X = jb.Fx;
    const long long nn = (long long)n * n;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < 3 * nn; i += (long long)gridDim.x * 256)
        X[i] = i >= 2 * nn && (i - 2 * nn) % (n + 1) == 0 ? 1.0 : 0.0;
}

__device__ __forceinline__ void live_slots(const MolState& s, int& newslot, unsigned& live_mask) {
    const int c = s.hist_count, head = s.hist_head;
    live_mask = 0;
    if (c < MAX_DIIS) {
        newslot = (head + c) % MAX_DIIS;
        for (int i = 0; i < c; ++i) live_mask |= 1u << ((head + i) % MAX_DIIS);
    } else {
        newslot = head;
        for (int i = 1; i < MAX_DIIS; ++i) live_mask |= 1u << ((head + i) % MAX_DIIS);
    }
}

constexpr int POST_WARPS = 8;

__global__ void __launch_bounds__(32 * POST_WARPS) k_post_fock(const ChanJob* __restrict__ jobs, const MolDesc* __restrict__ mols,
                                                               const MolState* __restrict__ st, int nblk, int energy_only, int force,
                                                               const int* __restrict__ skip) {
    if (skip && *skip) return;
    const ChanJob jb = jobs[blockIdx.y];
    const MolState& s = st[jb.mol];
    if (!force && !s.active) return;
    const int n = jb.n;
    const int nb = red_blocks(n);
    if ((int)blockIdx.x >= nb) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int newslot = 0;
    unsigned live = 0;
    live_slots(s, newslot, live);
    const long long ls = packed_sym_len(n);
    double acc[RED_N];
#pragma unroll
    for (int k = 0; k < RED_N; ++k) acc[k] = 0.0;
    const bool adiis = jb.hD != nullptr;
    for (int r = blockIdx.x * POST_WARPS + warp; r < n; r += nb * POST_WARPS) {
        const double* Fr = jb.F + (long long)r * n;
        const double* Pr = jb.P + (long long)r * n;
        const double* Hr = jb.H + (long long)r * n;
        const long long rs = sym_row(r, n);
        for (int c = r + lane; c < n; c += 32) {
            const long long si = rs + (c - r);
            // the live history entries are loaded with F, P and H, before this element's stores, so
            // an element costs one round trip to memory
            double hf[MAX_DIIS], hd[MAX_DIIS];
#pragma unroll
            for (int j = 0; j < MAX_DIIS; ++j) {
                const bool ld = !energy_only && adiis && j != newslot && (live >> j & 1u);
                hf[j] = ld ? jb.hF[j * ls + si] : 0.0;
                hd[j] = ld ? jb.hD[j * ls + si] : 0.0;
            }
            const double f = Fr[c], p = Pr[c], hh = Hr[c];
            const double wgt = c == r ? 1.0 : 2.0;
            acc[RED_E_H] += wgt * p * hh;
            acc[RED_E_F] += wgt * p * f;
            if (energy_only) continue;
            jb.hF[newslot * ls + si] = f;
            if (adiis) {
                jb.hD[newslot * ls + si] = p;
#pragma unroll
                for (int j = 0; j < MAX_DIIS; ++j)  // unrolled: no dynamic index into acc
                    if (j == newslot) {
                        acc[RED_GROW + j] += wgt * p * f;
                    } else if (live >> j & 1u) {
                        acc[RED_GROW + j] += wgt * p * hf[j];
                        acc[RED_GCOL + j] += wgt * hd[j] * f;
                    }
            }
        }
    }
    __shared__ double part[POST_WARPS][RED_N];
#pragma unroll
    for (int k = 0; k < RED_N; ++k) {
        double v = acc[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) part[warp][k] = v;
    }
    __syncthreads();
    if (threadIdx.x < RED_N) {
        double v = 0.0;
        for (int w = 0; w < POST_WARPS; ++w) v += part[w][threadIdx.x];
        jb.red[(long long)blockIdx.x * RED_N + threadIdx.x] = v;
    }
}

// The DIIS error e = FP - (FP)^T of the new Fock matrix (scf.rs:531-544).  F and P are symmetric,
// so (FP)^T = P.F and e = F.P - P.F: tile (I, J) of e is F[I,:].P[:,J] - P[I,:].F[:,J], one
// pipelined FP64 tensor-core k-loop over both products, and e is antisymmetric, so only the
// upper-triangle tiles are computed.  The epilogue takes the strict upper triangle: it stores e in
// the packed history slot of this iteration and forms this tile's share of |e|_F^2 and of
// <e, e_slot> for every live slot (the new CDIIS Gram row).
//
// COPY: how the operands reach shared memory: 0 8-byte cp.async, 1 16-byte cp.async (even n, 16-byte
// aligned rows), 2 tensor-memory-accelerator boxes from the job's tensor maps of F and P
// (maps[4 job + 2], maps[4 job + 3]; a copy wait that runs out sets bit 11 of *err).
constexpr int CT_LD = DG_TILE + 1;  // row stride of the staged commutator tile (doubles)

template <int COPY>
__device__ __forceinline__ void commutator_body(const ChanJob* __restrict__ jobs, const GemmTile* __restrict__ tiles, int t,
                                                const MolState* __restrict__ st, const TmaDesc* __restrict__ maps, int* __restrict__ err,
                                                double red[CP_N][4]) {
    const GemmTile tl = tiles[t];
    const ChanJob jb = jobs[tl.job];
    const MolState& s = st[jb.mol];
    if (!s.active) return;
    const int n = jb.n;
    int newslot = 0;
    unsigned live = 0;
    live_slots(s, newslot, live);
    const long long la = packed_anti_len(n);
    const int m0 = tl.tm * DG_TILE, n0 = tl.tn * DG_TILE;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // e is antisymmetric: a warp whose quarter is padding or lies below the diagonal issues no MMAs
    const bool compute = dg_quarter_on(m0, n0, n, n, tl.tm == tl.tn);
    double acc[2][4][4];
    double* T;  // the tile staged for the epilogue, in the pipeline's shared memory (free after the k-loop)
    if constexpr (COPY == 2) {
        extern __shared__ __align__(16) unsigned char ctsm[];
        __shared__ DtBars bars;
        const TmaDesc* mp = maps + 4 * tl.job;  // F and P are symmetric: B = F or P read by rows
        const int shape = dg_quarter_shape(m0, n0, n, n, tl.tm == tl.tn);
        if (!dg_mainloop_tma(dt_stages(ctsm), bars, mp + 2, mp + 3, mp + 3, mp + 2, false, n, m0, n0, acc, shape)) {
            if (threadIdx.x == 0) atomicOr(err, 1 << 11);
            return;
        }
        T = reinterpret_cast<double*>(dt_stages(ctsm));
    } else {
        extern __shared__ __align__(16) double dsm[];
        dg_mainloop_diff<COPY == 1>(dsm, jb.F, jb.P, jb.P, jb.F, n, n, m0, n0, acc, compute);
        T = dsm;
    }
    // e by tile rows: the strict upper triangle of a row is contiguous in the packed history, so each
    // warp's stores of e and loads of the live slots' error vectors are runs of consecutive words
    if (compute) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) T[dg_row(i, e) * CT_LD + dg_col(j, e)] = acc[i][j][e];
    }
    __syncthreads();
    double v[CP_N];
#pragma unroll
    for (int k = 0; k < CP_N; ++k) v[k] = 0.0;
    for (int rl = warp; rl < DG_TILE; rl += DG_THREADS / 32) {
        const int r = m0 + rl;
        if (r >= n) break;
        const long long arow = anti_row(r, n) - r - 1;  // packed index of (r, c) is arow + c
        // both columns' loads of the live slots before the row's stores: one round trip per row
        double eq[2][MAX_DIIS];
#pragma unroll
        for (int hlf = 0; hlf < 2; ++hlf) {
            const int c = n0 + lane + 32 * hlf;
            const bool in = r < c && c < n;
#pragma unroll
            for (int q = 0; q < MAX_DIIS; ++q)
                eq[hlf][q] = in && q != newslot && (live >> q & 1u) ? jb.hE[q * la + arow + c] : 0.0;
        }
#pragma unroll
        for (int hlf = 0; hlf < 2; ++hlf) {
            const int cl = lane + 32 * hlf, c = n0 + cl;
            if (r < c && c < n) {
                const double ev = T[rl * CT_LD + cl];
                const long long ai = arow + c;
                jb.hE[newslot * la + ai] = ev;
                v[CP_ERR2] += 2.0 * ev * ev;
#pragma unroll
                for (int q = 0; q < MAX_DIIS; ++q)
                    if (q == newslot)
                        v[CP_B + q] += ev * ev;
                    else if (live >> q & 1u)
                        v[CP_B + q] += ev * eq[hlf][q];
            }
        }
    }
#pragma unroll
    for (int k = 0; k < CP_N; ++k) {
        double x = v[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (lane == 0) red[k][warp] = x;
    }
    __syncthreads();
    if (tid < CP_N) {
        // index of tile (tm, tn), tm <= tn, in the channel's row-major upper-triangle tile list
        const int nt = (n + DG_TILE - 1) / DG_TILE;
        const int local = tl.tm * nt - tl.tm * (tl.tm - 1) / 2 + (tl.tn - tl.tm);
        jb.cpart[(long long)local * CP_N + tid] = red[tid][0] + red[tid][1] + red[tid][2] + red[tid][3];
    }
}

__global__ void __launch_bounds__(DG_THREADS, 4) k_commutator16(const ChanJob* __restrict__ jobs, const GemmTile* __restrict__ tiles,
                                                                int ntiles, const MolState* __restrict__ st) {
    __shared__ double red[CP_N][4];
    if ((int)blockIdx.x < ntiles) commutator_body<1>(jobs, tiles, (int)blockIdx.x, st, nullptr, nullptr, red);
}
__global__ void __launch_bounds__(DG_THREADS, 4) k_commutator8(const ChanJob* __restrict__ jobs, const GemmTile* __restrict__ tiles,
                                                               int ntiles, const MolState* __restrict__ st) {
    __shared__ double red[CP_N][4];
    if ((int)blockIdx.x < ntiles) commutator_body<0>(jobs, tiles, (int)blockIdx.x, st, nullptr, nullptr, red);
}
__global__ void __launch_bounds__(DG_THREADS, 4) k_commutator_tma(const ChanJob* __restrict__ jobs, const GemmTile* __restrict__ tiles,
                                                                  int ntiles, const MolState* __restrict__ st,
                                                                  const TmaDesc* __restrict__ maps, int* __restrict__ err) {
    __shared__ double red[CP_N][4];
    if ((int)blockIdx.x < ntiles) commutator_body<2>(jobs, tiles, (int)blockIdx.x, st, maps, err, red);
}
// The first nother CTAs take the tiles of odd n, as k_commutator8 (k_sp2_step_both says why).
__global__ void __launch_bounds__(DG_THREADS, 4) k_commutator_both(const ChanJob* __restrict__ jobs, const GemmTile* __restrict__ tiles,
                                                                   int ntiles, const GemmTile* __restrict__ other, int nother,
                                                                   const MolState* __restrict__ st,
                                                                   const TmaDesc* __restrict__ maps, int* __restrict__ err) {
    __shared__ double red[CP_N][4];
    const int t = (int)blockIdx.x - nother;
    if (t < 0) commutator_body<0>(jobs, other, (int)blockIdx.x, st, nullptr, nullptr, red);
    else if (t < ntiles) commutator_body<2>(jobs, tiles, t, st, maps, err, red);
}

// ---- the extrapolation, a warp per molecule.  The kernel is a handful of tiny dense problems behind
// one long list of partial sums, so it is bound by latency: one thread per molecule walked the list (a
// memory round trip every few entries) and worked on arrays in local memory.  Here lane k sums quantity k,
// the list's loads batched ahead of the adds, and the small problems run over the lanes in shared memory
// and registers.  Every sum keeps its order and every element its expression, so the bits are those of
// the one-thread form.  Measured: 676 -> 74 us on a 3072-orbital molecule, 38 -> 10 us on 32 waters, 18 ->
// 10 us on methane.
constexpr int DIIS_DIM = MAX_DIIS + 1;

struct DiisWarp {  // one warp's shared memory
    double tot[RED_N];
    double bm[MAX_DIIS * MAX_DIIS], gm[MAX_DIIS * MAX_DIIS];  // the Gram matrices, logical order
    double B[DIIS_DIM * DIIS_DIM], rhs[DIIS_DIM], x[DIIS_DIM];
};

// Gaussian elimination with partial pivoting on w.B (n x n, n <= DIIS_DIM) and w.rhs, a lane per row;
// false when a pivot is below 1e-12.  The solution is in w.x.
__device__ __forceinline__ bool solve_small(int n, DiisWarp& w, int lane) {
    double* m = w.B;
    double* rhs = w.rhs;
    for (int col = 0; col < n; ++col) {
        int piv = col;
        double best = fabs(m[col * n + col]);
        for (int row = col + 1; row < n; ++row) {
            const double v = fabs(m[row * n + col]);
            if (v > best) {
                best = v;
                piv = row;
            }
        }
        if (best < 1.0e-12) return false;
        __syncwarp();
        if (piv != col) {
            if (lane < n) {
                const double t = m[col * n + lane];
                m[col * n + lane] = m[piv * n + lane];
                m[piv * n + lane] = t;
            } else if (lane == 31) {
                const double t = rhs[col];
                rhs[col] = rhs[piv];
                rhs[piv] = t;
            }
            __syncwarp();
        }
        const int row = col + 1 + lane;
        if (row < n) {
            const double factor = m[row * n + col] / m[col * n + col];
            if (factor != 0.0) {
                for (int j = col; j < n; ++j) m[row * n + j] -= factor * m[col * n + j];
                rhs[row] -= factor * rhs[col];
            }
        }
        __syncwarp();
    }
    if (lane == 0)
        for (int col = n - 1; col >= 0; --col) {
            double sum = rhs[col];
            for (int j = col + 1; j < n; ++j) sum -= m[col * n + j] * w.x[j];
            w.x[col] = sum / m[col * n + col];
        }
    __syncwarp();
    return true;
}

// A-DIIS: projected gradient on the probability simplex (the Euclidean projection: sort descending,
// running threshold) for f(c) = 2 d.c + c.S c from c = e_m.  Lane k holds row k of S + S^T; every lane
// holds all of c.  The sort is a network on registers (entries past m are -inf and stay last) and the
// threshold's divisions run a lane per rank.
__device__ __forceinline__ void adiis_simplex(int m, double dk, const double (&Sk)[MAX_DIIS], double (&c)[MAX_DIIS], int lane) {
    constexpr unsigned ALL = 0xffffffffu;
    double L = 1.0e-12;
    {
        double row = 0.0;
#pragma unroll
        for (int j = 0; j < MAX_DIIS; ++j)
            if (j < m) row += fabs(Sk[j]);
#pragma unroll
        for (int i = 0; i < MAX_DIIS; ++i) {
            const double r = __shfl_sync(ALL, row, i);
            if (i < m) L = fmax(L, r);
        }
    }
    const double lr = 1.0 / L;
    const double ninf = __longlong_as_double(0xfff0000000000000LL);
    double ck = lane == m - 1 ? 1.0 : 0.0;  // this lane's own entry of c
#pragma unroll
    for (int i = 0; i < MAX_DIIS; ++i) c[i] = i == m - 1 ? 1.0 : 0.0;
    for (int it = 0; it < 400; ++it) {
        double acc = 2.0 * dk;
#pragma unroll
        for (int j = 0; j < MAX_DIIS; ++j)
            if (j < m) acc += Sk[j] * c[j];
        const double trial = ck - lr * acc;
        double v[MAX_DIIS], u[MAX_DIIS];
#pragma unroll
        for (int i = 0; i < MAX_DIIS; ++i) {
            v[i] = __shfl_sync(ALL, trial, i);
            u[i] = i < m ? v[i] : ninf;
        }
        // Batcher's odd-even merge sort of eight, descending
        auto cx = [&](int a, int b) {
            const bool sw = u[a] < u[b];
            const double hi = sw ? u[b] : u[a], lo = sw ? u[a] : u[b];
            u[a] = hi;
            u[b] = lo;
        };
        cx(0, 1); cx(2, 3); cx(4, 5); cx(6, 7);
        cx(0, 2); cx(1, 3); cx(4, 6); cx(5, 7);
        cx(1, 2); cx(5, 6);
        cx(0, 4); cx(1, 5); cx(2, 6); cx(3, 7);
        cx(2, 4); cx(3, 5);
        cx(1, 2); cx(3, 4); cx(5, 6);
        double css = 0.0, mine = 0.0, uj = 0.0;
#pragma unroll
        for (int j = 0; j < MAX_DIIS; ++j) {
            if (j < m) css += u[j];
            if (j == lane) {
                mine = css;
                uj = u[j];
            }
        }
        const double t = (mine - 1.0) / ((double)lane + 1.0);
        const unsigned on = __ballot_sync(ALL, lane < m && uj - t > 0.0);
        const double theta = on ? __shfl_sync(ALL, t, 31 - __clz(on)) : 0.0;
        double delta = 0.0;
#pragma unroll
        for (int i = 0; i < MAX_DIIS; ++i)
            if (i < m) {
                const double p = fmax(v[i] - theta, 0.0);
                delta += fabs(p - c[i]);
                c[i] = p;
            }
        ck = fmax(trial - theta, 0.0);
        if (delta < 1.0e-12) break;  // the same in every lane
    }
}

// Adds `count` values of a list to t in order: p[k * stride], SUM_BATCH loads ahead of their adds.
constexpr int SUM_BATCH = 16;
__device__ __forceinline__ double ordered_sum(double t, const double* __restrict__ p, int stride, int count) {
    for (int k0 = 0; k0 < count; k0 += SUM_BATCH) {
        double v[SUM_BATCH];
#pragma unroll
        for (int u = 0; u < SUM_BATCH; ++u) v[u] = k0 + u < count ? __ldcg(p + (long long)(k0 + u) * stride) : 0.0;
#pragma unroll
        for (int u = 0; u < SUM_BATCH; ++u)
            if (k0 + u < count) t += v[u];
    }
    return t;
}

__global__ void __launch_bounds__(32 * SCF_MOL_WARPS) k_diis_solve(const MolDesc* __restrict__ mols, const ChanJob* __restrict__ jobs,
                                                                   const int* __restrict__ mol_job0, int nmol, MolState* __restrict__ st,
                                                                   int* __restrict__ mol_status, int nblk, ScfParams prm) {
    __shared__ DiisWarp sh[SCF_MOL_WARPS];
    const int lane = threadIdx.x & 31, mi = blockIdx.x * SCF_MOL_WARPS + (threadIdx.x >> 5);
    if (mi >= nmol) return;
    MolState& s = st[mi];
    if (!s.active) return;
    DiisWarp& w = sh[threadIdx.x >> 5];
    const int nch = mols[mi].nch, job0 = mol_job0[mi];
    {
        double t = 0.0;
        for (int c = 0; c < nch; ++c) {
            const ChanJob& jb = jobs[job0 + c];
            if (lane < RED_N) t = ordered_sum(t, jb.red + lane, RED_N, red_blocks(jb.n));
            // the commutator pass, in tile order: CP_ERR2 into RED_ERR2, CP_B + k into RED_B + k
            static_assert(RED_B == RED_ERR2 + 1 && CP_B == CP_ERR2 + 1, "one lane per commutator sum");
            if (lane >= RED_ERR2 && lane < RED_ERR2 + CP_N) t = ordered_sum(t, jb.cpart + (lane - RED_ERR2), CP_N, jb.ntiles);
        }
        if (lane < RED_N) w.tot[lane] = t;
    }
    for (int i = lane; i < MAX_DIIS * MAX_DIIS; i += 32) {
        w.bm[i] = s.bmat[i];
        w.gm[i] = s.gmat[i];
    }
    // history bookkeeping: physical slot of logical index i is (head + i) % 8
    const int cnt = s.hist_count;
    int newslot, head = s.hist_head;
    unsigned live;
    live_slots(s, newslot, live);
    __syncwarp();
    const double* tot = w.tot;
    const double e_elec = 0.5 * (tot[RED_E_H] + tot[RED_E_F]);
    const double err = sqrt(tot[RED_ERR2]);
    if (cnt == MAX_DIIS) {  // drop the oldest: shift the Gram matrices up-left
        double b2[2], g2[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int e = lane + 32 * u, i = e / MAX_DIIS, j = e % MAX_DIIS;
            const bool in = i < MAX_DIIS - 1 && j < MAX_DIIS - 1;
            b2[u] = w.bm[in ? e + MAX_DIIS + 1 : e];
            g2[u] = w.gm[in ? e + MAX_DIIS + 1 : e];
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            w.bm[lane + 32 * u] = b2[u];
            w.gm[lane + 32 * u] = g2[u];
        }
        head = (head + 1) % MAX_DIIS;
        __syncwarp();
    }
    const int m = cnt == MAX_DIIS ? MAX_DIIS : cnt + 1, last = m - 1;
    if (lane < m) {
        const int phys = (head + lane) % MAX_DIIS;
        const double b = 2.0 * tot[RED_B + phys];
        w.bm[last * MAX_DIIS + lane] = b;
        w.bm[lane * MAX_DIIS + last] = b;
        if (lane != last) {
            w.gm[last * MAX_DIIS + lane] = tot[RED_GROW + phys];  // <D_last, F_i>
            w.gm[lane * MAX_DIIS + last] = tot[RED_GCOL + phys];  // <D_i, F_last>
        } else {
            w.gm[last * MAX_DIIS + last] = tot[RED_GROW + newslot];
        }
    }
    __syncwarp();
    for (int i = lane; i < MAX_DIIS * MAX_DIIS; i += 32) {
        s.bmat[i] = w.bm[i];
        s.gmat[i] = w.gm[i];
    }
    const bool diverged = !isfinite(e_elec) || !isfinite(err);
    if (lane == 0) {
        s.hist_head = head;
        s.hist_count = m;
        s.e_elec = e_elec;
        s.err_norm = err;
        s.mode = 0;
        s.accel_used = 0;
        if (diverged) {
            s.status = 4;  // AM1GPU_SCF_DIVERGED
            mol_status[mi] = 4;
            s.active = 0;
            s.iter += 1;
        }
    }
    if (diverged) return;
    int accel = prm.use_diis ? prm.accelerator : 0;
    if (nch == 2) accel = prm.use_diis ? 1 : 0;  // UHF: CDIIS only (scf.rs:770-803)
    bool use_adiis = accel == 2 && err > prm.adiis_switch;
    if (accel == 1 || (accel == 2 && !use_adiis)) {
        if (m >= 2) {
            const int dim = m + 1;
            for (int e = lane; e < dim * dim; e += 32) {
                const int i = e / dim, j = e % dim;
                w.B[e] = i < m && j < m ? w.bm[i * MAX_DIIS + j] : i == j ? 0.0 : -1.0;
            }
            if (lane < dim) w.rhs[lane] = lane == m ? -1.0 : 0.0;
            __syncwarp();
            if (solve_small(dim, w, lane)) {
                double wsum = 0.0;
                bool fin = true;
                for (int i = 0; i < m; ++i) {
                    wsum += fabs(w.x[i]);
                    fin = fin && isfinite(w.x[i]);
                }
                if (isfinite(wsum) && fin) {
                    if (lane < m) s.coeff[lane] = w.x[lane];
                    if (lane == 0) {
                        s.mode = 1;
                        s.accel_used = 1;
                    }
                }
            }
        }
    } else if (use_adiis && m >= 2) {
        const double gll = w.gm[last * MAX_DIIS + last];
        double Sk[MAX_DIIS], c[MAX_DIIS], dk = 0.0;
        bool fin = true;
#pragma unroll
        for (int j = 0; j < MAX_DIIS; ++j) Sk[j] = 0.0;
        if (lane < m) {
            const int k = lane;
            dk = w.gm[k * MAX_DIIS + last] - gll;
            fin = isfinite(dk);
#pragma unroll
            for (int j = 0; j < MAX_DIIS; ++j)
                if (j < m) {
                    const double skj = w.gm[k * MAX_DIIS + j] - w.gm[k * MAX_DIIS + last] - w.gm[last * MAX_DIIS + j] + gll;
                    const double sjk = w.gm[j * MAX_DIIS + k] - w.gm[j * MAX_DIIS + last] - w.gm[last * MAX_DIIS + k] + gll;
                    Sk[j] = skj + sjk;
                    fin = fin && isfinite(Sk[j]);
                }
        }
        // a Gram matrix that is not finite has no simplex minimum: plain F (energy and error are finite
        // here, so this takes an overflow in the products of two histories)
        if (__all_sync(0xffffffffu, fin)) {
            adiis_simplex(m, dk, Sk, c, lane);
#pragma unroll
            for (int i = 0; i < MAX_DIIS; ++i)
                if (i < m) {
                    fin = fin && isfinite(c[i]);
                }
            if (fin) {  // c is the same in every lane
#pragma unroll
                for (int i = 0; i < MAX_DIIS; ++i)
                    if (i < m && lane == i) s.coeff[i] = c[i];
                if (lane == 0) {
                    s.mode = 1;
                    s.accel_used = 2;
                }
            }
        }
    }
}

constexpr int COMBINE_CHUNK = 8;
constexpr double COMBINE_DIFF_GATE = 0.5;

__global__ void k_combine(const ChanJob* __restrict__ jobs, const MolState* __restrict__ st, int force) {
    const ChanJob jb = jobs[blockIdx.y];
    const MolState& s = st[jb.mol];
    if (!force && !s.active) return;
    const int n = jb.n;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const long long ls = packed_sym_len(n);
    const int m = s.hist_count;
    // from the second iteration on, F* still holds the previous iteration's: the distance between the
    // two (row sums of squares) lets k_sp2_bounds widen the previous spectral interval instead of
    // running the Lanczos bounds again.  It is only worth its extra read of F* once the density has
    // nearly settled (||P - P_previous||_F < COMBINE_DIFF_GATE); before that the rows report NaN and
    // the bounds run Lanczos.
    const bool diff = s.iter > 0 && s.dp * n < COMBINE_DIFF_GATE;
    const int mode = s.mode;
    const double* hrow[MAX_DIIS];  // history entries in logical order, and their coefficients
    double cf[MAX_DIIS];
#pragma unroll
    for (int i = 0; i < MAX_DIIS; ++i) {
        hrow[i] = jb.hF + ((s.hist_head + i) % MAX_DIIS) * ls;
        cf[i] = i < m ? s.coeff[i] : 0.0;
    }
    for (int r = blockIdx.x * nw + warp; r < n; r += gridDim.x * nw) {
        double* out = jb.Fx + (long long)r * n;
        double bound = 0.0, diag = 0.0, dd = 0.0;
        // chunks of COMBINE_CHUNK columns per lane: every load of a chunk (history entries, the previous
        // F*) is issued before any of its stores; each lane still visits its columns in ascending order
        for (int c0 = 0; c0 < n; c0 += 32 * COMBINE_CHUNK) {
            double val[COMBINE_CHUNK];
#pragma unroll
            for (int u = 0; u < COMBINE_CHUNK; ++u) {
                const int c = c0 + 32 * u + lane;
                double v = 0.0;
                if (c < n) {
                    if (mode == 0) {
                        v = jb.F[(long long)r * n + c];
                    } else {
                        const int lo = min(r, c), hi = max(r, c);
                        const long long si = sym_row(lo, n) + (hi - lo);
#pragma unroll
                        for (int i = 0; i < MAX_DIIS; ++i)
                            if (i < m) v += cf[i] * hrow[i][si];
                    }
                    if (diff) {
                        const double d = v - out[c];
                        dd = fma(d, d, dd);
                    }
                }
                val[u] = v;
            }
#pragma unroll
            for (int u = 0; u < COMBINE_CHUNK; ++u) {
                const int c = c0 + 32 * u + lane;
                if (c < n) {
                    out[c] = val[u];
                    if (c == r) diag = val[u];
                    else bound += fabs(val[u]);
                }
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            bound += __shfl_xor_sync(0xffffffffu, bound, o);
            diag += __shfl_xor_sync(0xffffffffu, diag, o);
            dd += __shfl_xor_sync(0xffffffffu, dd, o);
        }
        if (lane == 0) {
            jb.rowmin[r] = diag - bound;
            jb.rowmax[r] = diag + bound;
            jb.rowdf[r] = diff ? dd : __longlong_as_double(0x7ff8000000000000LL);
        }
    }
}

__global__ void k_density_post(const ChanJob* __restrict__ jobs, const MolState* __restrict__ st, int nblk, const int* __restrict__ mask,
                               int want) {
    const ChanJob jb = jobs[blockIdx.y];
    if (!st[jb.mol].active || (mask && (mask[jb.mol] != 0) != (want != 0))) return;
    const int nb = dens_blocks(jb.n);
    if ((int)blockIdx.x >= nb) return;
    const long long nn = (long long)jb.n * jb.n;
    double acc = 0.0;
    const long long stride = (long long)nb * blockDim.x;
    // four elements per trip, their loads before their stores; each thread keeps its order of the sum
    for (long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x; i0 < nn; i0 += 4 * stride) {
        double pn[4], po[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const long long i = i0 + u * stride;
            pn[u] = i < nn ? jb.Pnew[i] : 0.0;
            po[u] = i < nn ? jb.P[i] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const long long i = i0 + u * stride;
            if (i >= nn) break;
            const double d = pn[u] - po[u];
            acc += d * d;
            jb.P[i] = pn[u];
        }
    }
    __shared__ double part[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) part[warp] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double v = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v += part[w];
        jb.red2[blockIdx.x] = v;
    }
}

// A warp per molecule: its lanes fetch the partial sums, 32 blocks of a channel at a time, every lane
// adds them in block order, and lane 0 takes the decision.
__global__ void __launch_bounds__(32 * SCF_MOL_WARPS) k_converge(const MolDesc* __restrict__ mols, const ChanJob* __restrict__ jobs,
                                                                 const int* __restrict__ mol_job0, int nmol, MolState* __restrict__ st,
                                                                 int* __restrict__ mol_status, int nblk, ScfParams prm,
                                                                 int* __restrict__ active_count, const int* __restrict__ mask, int want) {
    const int lane = threadIdx.x & 31, mi = blockIdx.x * SCF_MOL_WARPS + (threadIdx.x >> 5);
    if (mi >= nmol) return;
    MolState& s = st[mi];
    if (!s.active || (mask && (mask[mi] != 0) != (want != 0))) return;
    if (mol_status[mi] != 0) {  // the eigensolver refused its input
        __syncwarp();
        if (lane == 0) {
            s.active = 0;
            s.status = mol_status[mi];
            s.iter += 1;
        }
        return;
    }
    const int nch = mols[mi].nch, job0 = mol_job0[mi];
    double dp = 0.0;
    for (int c = 0; c < nch; ++c) {
        const ChanJob& jb = jobs[job0 + c];
        const int nb = dens_blocks(jb.n);
        double ss = 0.0;
        for (int b0 = 0; b0 < nb; b0 += 32) {
            const double v = b0 + lane < nb ? __ldcg(jb.red2 + b0 + lane) : 0.0;
            for (int b = 0; b < min(32, nb - b0); ++b) ss += __shfl_sync(0xffffffffu, v, b);
        }
        dp += sqrt(ss / fmax((double)jb.n * jb.n, 1.0));
    }
    if (lane != 0) return;
    const double de = fabs(s.e_elec - s.e_old);
    s.dp = dp;
    s.e_old = s.e_elec;
    s.residual = s.err_norm;
    const int it = s.iter;
    s.iter = it + 1;
    if (s.lowp) {
        // mixed precision: this iteration's density came from TF32 purification, so no
        // convergence is declared on it; the TF32 phase ends once the density has settled near its
        // rounding level, and the FP64 iterations that follow take the SCF to convergence
        if ((it > 0 && dp < prm.lowp_switch) || s.iter >= prm.lowp_max_iter) {
            s.lowp = 0;
            s.lowp_end = it;
            s.lowp_flush = 1;
        }
        if (s.iter >= prm.max_scf) s.active = 0;
    } else if (s.lowp_flush) {
        // first FP64 iteration: its Fock matrix was built from the last TF32 density.  The
        // history restarts after it, so the extrapolation (A-DIIS in particular, whose energy
        // model would favour that slightly non-idempotent density) sees FP64 iterations only.
        s.lowp_flush = 0;
        s.hist_count = 0;
        if (s.iter >= prm.max_scf) s.active = 0;
    } else if (it > s.lowp_end && it > 0 && de < prm.e_tol && (dp < prm.p_tol || s.err_norm < 1.0e-7)) {
        s.converged = 1;
        s.active = 0;
    } else if (s.iter >= prm.max_scf) {
        s.active = 0;
    }
    if (s.active) {
        atomicAdd(active_count, 1);
        if (s.lowp) atomicAdd(active_count + 1, 1);
    }
}

// A warp per molecule: lanes 0 and 1 add the two energy traces, in block order.
__global__ void __launch_bounds__(32 * SCF_MOL_WARPS) k_final_energy(const MolDesc* __restrict__ mols, const ChanJob* __restrict__ jobs,
                                                                     const int* __restrict__ mol_job0, int nmol,
                                                                     MolState* __restrict__ st, int nblk, const int* __restrict__ skip) {
    const int lane = threadIdx.x & 31, mi = blockIdx.x * SCF_MOL_WARPS + (threadIdx.x >> 5);
    if (mi >= nmol || (skip && *skip)) return;
    const int nch = mols[mi].nch, job0 = mol_job0[mi];
    double t = 0.0;
    for (int c = 0; c < nch; ++c) {
        const ChanJob& jb = jobs[job0 + c];
        if (lane < 2) t = ordered_sum(t, jb.red + (lane == 0 ? RED_E_H : RED_E_F), RED_N, red_blocks(jb.n));
    }
    const double ef = __shfl_sync(0xffffffffu, t, 1);
    if (lane == 0) st[mi].e_final = 0.5 * (t + ef);
}

// Result record of one molecule (src/scf.rs:370-438): energies, heat of formation, Mulliken
// charges, dipole (point charges + s-p hybrid term), frontier orbitals.  A CTA per molecule, a thread
// per atom (the sums over atoms: thread-strided, then a fixed tree, so they depend on the molecule alone).
// One thread per molecule cost a chain of memory round trips per atom: 1956 us for 1536 atoms, now 37 us.
__global__ void __launch_bounds__(RESULT_THREADS) k_results(const MolDesc* __restrict__ mols, const ChanJob* __restrict__ jobs,
                                                            const int* __restrict__ mol_job0, int nmol, const MolState* __restrict__ st,
                                                            const int* __restrict__ mol_status, const DevElem* __restrict__ params,
                                                            const int* __restrict__ atom_z, const double* __restrict__ atom_xyz,
                                                            double* __restrict__ res, double* __restrict__ charges,
                                                            const int* __restrict__ skip) {
    __shared__ double part[5][RESULT_THREADS / 32];
    const int mi = blockIdx.x;
    if (mi >= nmol || (skip && *skip)) return;
    const MolDesc md = mols[mi];
    const MolState& s = st[mi];
    const int n = md.nao, h = md.nheavy, tid = threadIdx.x;
    const double* P0 = jobs[mol_job0[mi]].P;
    const double* P1 = md.nch == 2 ? jobs[mol_job0[mi] + 1].P : nullptr;
    double sum[5] = {0.0, 0.0, 0.0, 0.0, 0.0};  // e_isol, eheat, dipole
    for (int A = tid; A < md.natoms; A += RESULT_THREADS) {
        const int a = md.atom_base + A;
        const DevElem& e = params[md.method * (MAX_Z + 1) + atom_z[a]];
        sum[0] += e.e_isol;
        sum[1] += e.eheat_ev;
        const int o = A < h ? 4 * A : 4 * h + (A - h), no = A < h ? 4 : 1;
        double pop = 0.0;
        for (int k = 0; k < no; ++k) {
            const long long d = (long long)(o + k) * n + o + k;
            pop += P1 ? P0[d] + P1[d] : P0[d];
        }
        const double q = e.core_charge - pop;
        charges[a] = q;
        for (int k = 0; k < 3; ++k) sum[2 + k] += atom_xyz[3 * a + k] * q;
        if (e.norb == 4) {
            const double hyb = -2.0 * e.dd;
            for (int k = 0; k < 3; ++k) {
                const long long idx = (long long)o * n + o + 1 + k;
                sum[2 + k] += hyb * (P1 ? P0[idx] + P1[idx] : P0[idx]);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        double v = sum[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((tid & 31) == 0) part[k][tid >> 5] = v;
    }
    __syncthreads();
    if (tid != 0) return;
    for (int k = 0; k < 5; ++k) {
        sum[k] = part[k][0];
        for (int w = 1; w < RESULT_THREADS / 32; ++w) sum[k] += part[k][w];
    }
    const double e_isol = sum[0], eheat = sum[1];
    const double* dip = sum + 2;
    double* r = res + (long long)mi * RES_N;
    const double total = s.e_final + s.core_ev;
    r[RES_ELEC] = s.e_final;
    r[RES_CORE] = s.core_ev;
    r[RES_TOTAL] = total;
    r[RES_HOF] = (total - e_isol + eheat) * EV_TO_KCAL;
    double mag = 0.0;
    for (int k = 0; k < 3; ++k) {
        r[RES_DIP + k] = dip[k] * AU_DIPOLE_TO_DEBYE;
        mag += r[RES_DIP + k] * r[RES_DIP + k];
    }
    r[RES_DIPMAG] = sqrt(mag);
    const double nan = __longlong_as_double(0x7ff8000000000000LL);
    const double* ea = jobs[mol_job0[mi]].eps;
    const int na = md.n_occ[0], nb = md.n_occ[1];
    r[RES_HOMO] = na >= 1 ? ea[na - 1] : nan;
    r[RES_LUMO] = na < n ? ea[na] : nan;
    r[RES_HOMO_B] = nan;
    r[RES_LUMO_B] = nan;
    if (md.nch == 2) {
        const double* eb = jobs[mol_job0[mi] + 1].eps;
        r[RES_HOMO_B] = nb >= 1 ? eb[nb - 1] : nan;
        r[RES_LUMO_B] = nb < n ? eb[nb] : nan;
    }
    r[RES_RESID] = s.residual;
    r[RES_ITER] = (double)s.iter;
    r[RES_CONV] = (double)s.converged;
    r[RES_STATUS] = (double)(mol_status[mi] ? mol_status[mi] : s.status);
}

}  // namespace am1
