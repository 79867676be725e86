"""Orbital energies by a warp per eigenvalue (few of them) and by a thread per eigenvalue (many): the same bits."""

import numpy as np
import pytest

from am1gpu import _abi, workloads as W

pytestmark = pytest.mark.gpu


def _mol(kind, size, seed=3):
    rng = np.random.default_rng(seed)
    m = W.water_cluster(size, rng) if kind == "water" else W.alkane(size, rng, radical=kind == "radical")
    return (m.numbers, _abi.angstrom_to_bohr(m.xyz), 0.0, m.multiplicity)


def test_alone_equals_in_a_large_batch(gpu):
    mols = [_mol("alkane", 1), _mol("water", 1), _mol("alkane", 2), _mol("radical", 5), _mol("water", 20), _mol("alkane", 36), _mol("water", 75)]
    alone = [gpu.scf(*m, want_matrices=False) for m in mols]  # at most 450 eigenvalues a launch
    status, res = gpu.scf_batch(mols + [_mol("water", 1, k) for k in range(120)])  # 128 channels x 450 rows of a grid
    assert not any(status)
    for a, b in zip(alone, res):
        assert np.array_equal(a["mo_energies"], b["mo_energies"])
        assert np.all(np.diff(a["mo_energies"]) >= 0.0)
