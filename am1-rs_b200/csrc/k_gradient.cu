// Closed-form nuclear gradient of the NDDO energy at a fixed (converged) density: the
// Hellmann-Feynman gradient of am1-rs's closed_form_gradient (src/gradient.rs:173-253), i.e.
// fixed_density_gradient (src/gradient.rs:317-334) = the core-core gradient
// (src/repulsion.rs:81-115) + the electronic pair gradient (src/gradient.rs:366-493).
//
// Every term of the energy is a sum over atom pairs of a function of the pair displacement
// delta = x_b - x_a, so each pair contributes f = dE_pair/d(delta) to atom b and -f to atom a:
//   core-core        dE_cc(r)/d(delta)
//   resonance        sum_{mu in a, la in b} P_{mu la} (beta_mu + beta_la) dS_{mu la}
//   electron-core    sum_{mu nu in a} P_{mu nu} de1b_{mu nu} + sum_{la si in b} P_{la si} de2a_{la si}
//   two-electron     sum_{mu nu in a, la si in b} [P_{mu nu} P_{la si}
//                         - (Pa_{mu la} Pa_{nu si} + Pb_{mu la} Pb_{nu si})] d(mu nu|la si)
// with P the total density and Pa, Pb the spin densities (RHF: Pa = Pb = P/2, which gives the
// reference's -1/2 P_{mu la} P_{nu si}).  The derivatives are exact: the integral, overlap and
// core-core templates of integrals_t.cuh run on dual numbers, carrying d/dr where a quantity depends on the
// distance alone and d/d(delta) where it is turned into the molecule's frame.
//
// Each pair's f is formed once (k_pair_gradient) and a warp per atom adds its pairs' +-f, a pair per lane and then a
// fixed-order warp reduction (k_gradient): deterministic, no atomics.  The pair kernel is bound by FP64 latency
// at the eight warps of 255 registers an SM holds; what it does is the ten rows of a heavy-heavy pair's
// integrals (200 us for one pair by one thread).  So a warp holds pairs of one kind where it can: heavy-heavy first,
// then heavy-hydrogen, then hydrogen-hydrogen, molecule by molecule; few pairs are shared by four warps.  Before,
// each atom's warp evaluated its pairs, so every pair was evaluated twice, with three derivatives throughout: 192
// molecules of 79 atoms 3.08 -> 1.27 ms, C13H27 317 -> 120 us (whole pairs 208 us).  The two-centre integrals are contracted as they are
// formed (pair_integrals_each), so no block of 100 dual numbers is held per thread.
#include <cuda_runtime.h>

#include "am1gpu_internal.h"
#include "integrals_t.cuh"
#include "kernels.h"

namespace am1 {

// dE_pair/d(delta) of the pair (a, b) at fixed densities in parts, each handed to put(k, f): part 0 the core-core
// and resonance terms, parts 1 to 10 the rows of a heavy-heavy pair's integrals, part 1 all the integrals of any
// other pair; parts: those wanted, a bit each.  False for an element without the overlap (part 0).  Pa:
// channel-0 density (RHF: total), Pb: channel 1 or nullptr (RHF), both n x n in the internal AO order; oa, ob:
// first AO of a and b.
constexpr int GRAD_PARTS = 11;

template <class Put>
__device__ bool pair_force(const DevElem& ea, const DevElem& eb, int za, int zb, const double dl[3], const double* __restrict__ Pa,
                           const double* __restrict__ Pb, int n, int oa, int ob, unsigned parts, Put&& put) {
    const D3 dv[3] = {D3{dl[0], {1.0, 0.0, 0.0}}, D3{dl[1], {0.0, 1.0, 0.0}}, D3{dl[2], {0.0, 0.0, 1.0}}};
    const D1 r = D1{sqrt(dl[0] * dl[0] + dl[1] * dl[1] + dl[2] * dl[2]), {1.0}};
    double f[3] = {0.0, 0.0, 0.0};
    if (r.v < 1.0e-8) return true;  // coincident atoms: no direction, nothing to differentiate
    auto acc = [&](double c, const D3& x) {
        f[0] += c * x.d[0];
        f[1] += c * x.d[1];
        f[2] += c * x.d[2];
    };
    auto pt = [&](int r0, int c0) { return Pb ? Pa[(long long)r0 * n + c0] + Pb[(long long)r0 * n + c0] : Pa[(long long)r0 * n + c0]; };
    // exchange weight Pa Pa + Pb Pb (RHF: 2 (P/2)(P/2))
    auto px = [&](int r1, int c1, int r2, int c2) {
        const double x = Pa[(long long)r1 * n + c1] * Pa[(long long)r2 * n + c2];
        return Pb ? x + Pb[(long long)r1 * n + c1] * Pb[(long long)r2 * n + c2] : 0.5 * x;
    };
    const double u[3] = {dl[0] / r.v, dl[1] / r.v, dl[2] / r.v};
    const bool heavy = ea.norb == 4 && eb.norb == 4;
    if (parts & 1) {
        // core-core (src/repulsion.rs:81-115)
        acc(1.0, lift(pair_core_energy(ea, eb, za, zb, r), u));
        // resonance: H_{mu la} = (beta_mu + beta_la)/2 S_{mu la} in both triangles (src/gradient.rs:424-433)
        const D3 r3 = lift(r, u);
        const D3 dir[3] = {dv[0] / r3, dv[1] / r3, dv[2] / r3};
        D3 S[4][4];
        if (!overlap_block(ea, eb, r, dir, u, S)) return false;
        for (int i = 0; i < ea.norb; ++i) {
            const double bi = i == 0 ? ea.beta_s : ea.beta_p;
            for (int j = 0; j < eb.norb; ++j) acc(pt(oa + i, ob + j) * (bi + (j == 0 ? eb.beta_s : eb.beta_p)), S[i][j]);
        }
        put(0, f);
        f[0] = f[1] = f[2] = 0.0;
    }
    if (!(heavy ? parts >> 1 : parts & 2)) return true;
    // two-centre integrals, contracted as they are formed (no integral block is stored): the
    // element (kk ll | mm nn), kk >= ll on a and mm >= nn on b, stands for every ordering of its
    // index pairs (src/gradient.rs:434-466 sums over all of them):
    //   electron-core  e1b = -Z_b (mu nu | s s) on a's block, e2a = -Z_a (s s | la si) on b's
    //   Coulomb        P_{mu nu} P_{la si}
    //   exchange       -(Pa_{mu la} Pa_{nu si} + Pb_{mu la} Pb_{nu si})
    pair_integrals_each(ea, eb, dv, r, u, [=](int row) { return parts >> (row + 1) & 1; }, [&](int kk, int ll, int mm, int nn, const D3& v) {
        const int ma = kk == ll ? 1 : 2, mb = mm == nn ? 1 : 2;
        const double pa = pt(oa + kk, oa + ll), pb = pt(ob + mm, ob + nn);
        double c = ma * mb * pa * pb;
        c -= px(oa + kk, ob + mm, oa + ll, ob + nn);
        if (ll != kk) c -= px(oa + ll, ob + mm, oa + kk, ob + nn);
        if (nn != mm) {
            c -= px(oa + kk, ob + nn, oa + ll, ob + mm);
            if (ll != kk) c -= px(oa + ll, ob + nn, oa + kk, ob + mm);
        }
        if (mm == 0) c -= eb.core_charge * ma * pa;  // (kk ll | s s)
        if (kk == 0) c -= ea.core_charge * mb * pb;  // (s s | mm nn)
        acc(c, v);
        if (heavy && mm == 3 && nn == 3) {  // the row is complete
            put(1 + kk * (kk + 1) / 2 + ll, f);
            f[0] = f[1] = f[2] = 0.0;
        }
    });
    if (!heavy) put(1, f);
    return true;
}

// dE_pair/d(delta) of every pair of the batch.  A thread per pair, or (SPLIT) four warps to 32 pairs: one takes part 0,
// three take rows of about equal work.  Both add the parts in the same order, so they give the same bits.
template <bool SPLIT>
__device__ __forceinline__ void pair_gradient(const MolDesc* __restrict__ mols, int nmol, const long long* __restrict__ pair_prefix,
                                              long long npairs, const DevElem* __restrict__ params, const int* __restrict__ atom_z,
                                              const double* __restrict__ atom_xyz, const ChanJob* __restrict__ jobs,
                                              const int* __restrict__ mol_job0, double* __restrict__ pairf,
                                              int* __restrict__ mol_status) {
    const long long g0 = SPLIT ? blockIdx.x * 32LL + (threadIdx.x & 31) : (long long)blockIdx.x * GRAD_THREADS + threadIdx.x;
    if (!SPLIT && g0 >= npairs) return;
    const long long g = SPLIT ? min(g0, npairs - 1) : g0;  // a thread past the end repeats the last pair, for the barrier
    const int m = find_mol(pair_prefix, nmol, g);
    const MolDesc md = mols[m];
    // the pair (i < j): heavy atoms come first in the internal order, so i is the heavy one
    // whenever the pair mixes a heavy atom and a hydrogen (src/gradient.rs:394-401)
    int i, j;
    const int N = md.natoms, n = md.nao, h = md.nheavy, x = N - h;
    const int p = (int)(g - pair_prefix[m]), xx = h * (h - 1) / 2, xh = h * x;
    if (p < xx) pair_ij(p, h, i, j);
    else if (p < xx + xh) i = (p - xx) / x, j = h + (p - xx) % x;
    else pair_ij(p - xx - xh, x, i, j), i += h, j += h;
    const double* Pa = jobs[mol_job0[m]].P;
    const double* Pb = md.nch == 2 ? jobs[mol_job0[m] + 1].P : nullptr;
    const DevElem* tab = params + md.method * (MAX_Z + 1);
    const int ai = md.atom_base + i, aj = md.atom_base + j;
    const int zi = atom_z[ai], zj = atom_z[aj];
    const double dl[3] = {atom_xyz[3 * aj] - atom_xyz[3 * ai], atom_xyz[3 * aj + 1] - atom_xyz[3 * ai + 1],
                          atom_xyz[3 * aj + 2] - atom_xyz[3 * ai + 2]};
    const int oi = i < h ? 4 * i : 4 * h + (i - h), oj = j < h ? 4 * j : 4 * h + (j - h);
    double f[3] = {0.0, 0.0, 0.0};
    double* o = pairf + 3 * (md.pair_base + (long long)i * N - (long long)i * (i + 1) / 2 + (j - i - 1));
    if constexpr (SPLIT) {
        // rows (0 0) (1 0) (1 1) (2 1) | (2 0) (2 2) (3 1) | (3 0) (3 2) (3 3)
        constexpr unsigned kParts[4] = {1u, 0x17u << 1, 0xa8u << 1, 0x340u << 1};
        __shared__ double part[GRAD_PARTS][3][32];
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const unsigned mine = warp == 0 ? kParts[0] : warp == 1 ? kParts[1] : warp == 2 ? kParts[2] : kParts[3];
        for (int k = 0; k < GRAD_PARTS; ++k)
            if (mine >> k & 1)
                for (int c = 0; c < 3; ++c) part[k][c][lane] = 0.0;
        const bool ok = pair_force(tab[zi], tab[zj], zi, zj, dl, Pa, Pb, n, oi, oj, mine, [&](int k, const double* fk) {
            for (int c = 0; c < 3; ++c) part[k][c][lane] = fk[c];
        });
        if (!ok) atomicExch(&mol_status[m], 6);  // AM1GPU_UNSUPPORTED (also refused by the SCF itself)
        __syncthreads();
        if (warp > 0 || g0 >= npairs) return;
        for (int k = 0; k < GRAD_PARTS; ++k)
            for (int c = 0; c < 3; ++c) f[c] += part[k][c][lane];
    } else {
        const bool ok = pair_force(tab[zi], tab[zj], zi, zj, dl, Pa, Pb, n, oi, oj, (1u << GRAD_PARTS) - 1, [&](int, const double* fk) {
            for (int c = 0; c < 3; ++c) f[c] += fk[c];
        });
        if (!ok) atomicExch(&mol_status[m], 6);  // AM1GPU_UNSUPPORTED (also refused by the SCF itself)
    }
    o[0] = f[0];
    o[1] = f[1];
    o[2] = f[2];
}

#define AM1_PAIR_GRADIENT(NAME, THREADS, SPLIT)                                                                                      \
    __global__ void __launch_bounds__(THREADS)                                                                                       \
        NAME(const MolDesc* mols, int nmol, const long long* pair_prefix, long long npairs, const DevElem* params, const int* atom_z, \
             const double* atom_xyz, const ChanJob* jobs, const int* mol_job0, double* pairf, int* mol_status) {                      \
        pair_gradient<SPLIT>(mols, nmol, pair_prefix, npairs, params, atom_z, atom_xyz, jobs, mol_job0, pairf, mol_status);          \
    }
AM1_PAIR_GRADIENT(k_pair_gradient, GRAD_THREADS, false)
AM1_PAIR_GRADIENT(k_pair_gradient_split, 128, true)
#undef AM1_PAIR_GRADIENT

constexpr int GRAD_WARPS = 8;

// gradient[3 a + k] = dE/dx_{a,k} (eV/Bohr) for every atom of the batch, internal atom order.
__global__ void __launch_bounds__(32 * GRAD_WARPS) k_gradient(const MolDesc* __restrict__ mols, const int* __restrict__ atom_mol,
                                                              int natoms_total, const double* __restrict__ pairf,
                                                              double* __restrict__ gradient) {
    const int a = blockIdx.x * GRAD_WARPS + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (a >= natoms_total) return;  // uniform over the warp
    const MolDesc& md = mols[atom_mol[a]];
    const int A = a - md.atom_base, N = md.natoms;
    const double* pf = pairf + 3 * md.pair_base;
    double g[3] = {0.0, 0.0, 0.0};
    for (int B = lane; B < N; B += 32) {
        if (B == A) continue;
        const int i = min(A, B), j = max(A, B);
        const double* f = pf + 3 * ((long long)i * N - (long long)i * (i + 1) / 2 + (j - i - 1));
        const double sg = A == j ? 1.0 : -1.0;  // +f on the second atom of the pair, -f on the first
        g[0] += sg * f[0];
        g[1] += sg * f[1];
        g[2] += sg * f[2];
    }
    for (int o = 16; o > 0; o >>= 1) {
        g[0] += __shfl_xor_sync(0xffffffffu, g[0], o);
        g[1] += __shfl_xor_sync(0xffffffffu, g[1], o);
        g[2] += __shfl_xor_sync(0xffffffffu, g[2], o);
    }
    if (lane == 0) {
        gradient[3LL * a] = g[0];
        gradient[3LL * a + 1] = g[1];
        gradient[3LL * a + 2] = g[2];
    }
}

}  // namespace am1
