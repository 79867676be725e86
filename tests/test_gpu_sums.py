"""The per-channel and per-molecule sums at the edges of their blocks: the density-change and
purification-start blocks grow with the matrix from 512 orbitals on, and the purification's update
takes its tiles' partial sums 64 at a time (66 tiles at 642 orbitals)."""

import numpy as np
import pytest

from am1gpu import _abi, workloads as W

pytestmark = pytest.mark.gpu


def _water(k, seed=5):
    m = W.water_cluster(k, np.random.default_rng(seed))
    return (m.numbers, _abi.angstrom_to_bohr(m.xyz), 0.0, 1)


@pytest.mark.parametrize("k", [85, 86, 107])  # 510, 516 and 642 orbitals
def test_large_density_sums(gpu, k):
    mol, small = _water(k), _water(2)
    alone = gpu.scf(*mol, want_matrices=True)
    assert alone["status"] == 0 and alone["converged"]
    p, n = alone["density"], 6 * k
    # P/2 is the projector onto 4k of 6k orbitals.  The purification stops at its rounding floor, where
    # each product leaves at most n eps of error per element of a matrix of norm 1: n * 2.2e-16 * 2 (the
    # density's weight) with a factor 10 for the last steps
    tol = 20 * n * 2.2e-16
    assert abs(np.trace(p) - 8 * k) < tol * n
    assert np.max(np.abs(p @ p - 2.0 * p)) < 10 * tol
    assert abs(alone["charges"].sum()) < tol * n
    status, both = gpu.scf_batch([small, mol], want_matrices=True)
    assert list(status) == [0, 0]
    assert np.array_equal(both[1]["density"], p)
    assert both[1]["iterations"] == alone["iterations"]
    assert both[1]["energy_ev"] == alone["energy_ev"]
