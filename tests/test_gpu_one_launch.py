"""The one-launch purification (k_sp2_res, k_sp2_clu) at the edges of its tiles and paddings: against the
exact projector, and bit for bit against the launch-per-step kernels, which a batch with more than 16
channels of 113 to 448 orbitals takes."""

import numpy as np
import pytest

from am1gpu import _abi, workloads as W

pytestmark = pytest.mark.gpu


def _gapped(n, occ, seed):
    rng = np.random.default_rng(seed)
    eps = np.concatenate([rng.uniform(-40.0, -12.0, occ), rng.uniform(1.0, 10.0, n - occ)])
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    f = (q * eps) @ q.T
    return 0.5 * (f + f.T)


@pytest.mark.parametrize("n", [2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 72, 73, 79, 111, 112, 113, 127, 128, 129, 160,
                               191, 192, 193, 256, 257, 321, 384, 447, 448])
def test_projector(gpu, n):
    occ = max(1, (2 * n) // 3)
    f = _gapped(n, occ, n)
    p, steps = gpu.density_purify(f, occ)
    w, v = np.linalg.eigh(f)
    # the last squaring leaves n eps per element at norm 1, LAPACK's vectors n eps ||f|| / gap = 4 n eps; weight 2, a
    # factor 10 for the steps before the floor
    assert np.max(np.abs(p - 2.0 * v[:, :occ] @ v[:, :occ].T)) < 100 * max(n, 8) * 2.2e-16
    assert 0 < steps < 40
    assert np.array_equal(p, p.T)


MOLECULES = [("water", 19, 114), ("water", 32, 192), ("water", 43, 258), ("water", 74, 444), ("alkane", 21, 128),
             ("radical", 21, 127), ("radical", 40, 241)]


@pytest.mark.parametrize("kind,k,n", MOLECULES)
def test_alone_equals_in_a_batch(gpu, kind, k, n):
    def mol(kind, k, seed):
        m = W.water_cluster(k, np.random.default_rng(seed)) if kind == "water" else W.alkane(k, np.random.default_rng(seed),
                                                                                          radical=kind == "radical")
        return (m.numbers, _abi.angstrom_to_bohr(m.xyz), 0.0, m.multiplicity)

    m = mol(kind, k, 31)
    alone = gpu.scf(*m)
    assert alone["status"] == 0 and alone["nao"] == n
    status, res = gpu.scf_batch([mol("water", 20, 50 + i) for i in range(17)] + [m, mol("alkane", 3, 9)], want_matrices=True)
    assert all(x == 0 for x in status)
    r = res[17]
    assert np.array_equal(r["density"], alone["density"])
    assert r["iterations"] == alone["iterations"] and r["energy_ev"] == alone["energy_ev"]
