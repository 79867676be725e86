"""The reduction to tridiagonal form on the whole GPU below 2048 rows (a lone matrix leaves the cluster at
about 650 rows; panels of 32, so remainders of 1, 31 and 32 columns), and the bisection's two forms: a warp per
eigenvalue for few of them, a thread per eigenvalue for many, the same bits."""

import numpy as np
import pytest

from am1gpu import _abi, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [640, 672, 673, 703, 705, 1001, 1501, 2047])
def test_lone_matrix(gpu, n):
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n)) * (4.0 / np.sqrt(n))
    a = 0.5 * (a + a.T)
    a[np.diag_indices(n)] += rng.uniform(-40.0, 10.0, n)
    w, v = gpu.eigh(a)
    nrm = np.max(np.abs(w))
    # backward stable reduction, bisection and back-transformation: n eps ||A||, factor 10 for the constants
    tol = 10 * n * 2.2e-16
    assert np.max(np.abs(w - np.linalg.eigvalsh(a))) < tol * nrm
    assert np.max(np.abs(a @ v - v * w)) < tol * nrm
    assert np.max(np.abs(v.T @ v - np.eye(n))) < 1e-10  # inverse iteration outside clusters: eps / 1e-4
    assert np.array_equal(gpu.eigvalsh(a), w)


def test_eigenvalues_alone_and_among_many(gpu):
    def mol(m):
        return (m.numbers, _abi.angstrom_to_bohr(m.xyz), 0.0, m.multiplicity)

    big = mol(W.water_cluster(20, np.random.default_rng(1)))  # 120 orbitals
    alone = gpu.scf(*big, want_matrices=False)
    fill = [mol(W.alkane(1, np.random.default_rng(i))) for i in range(400)]  # 401 x 120 eigenvalues' warps: past four waves
    status, res = gpu.scf_batch([big] + fill)
    assert all(x == 0 for x in status)
    assert np.array_equal(res[0]["mo_energies"], alone["mo_energies"])
