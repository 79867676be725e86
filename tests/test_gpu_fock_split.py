"""The exchange blocks of k_fock on warps of their own (launches of fewer than 32768 atoms) and on the
atom's warp (more): the same bits, at the edges of a chunk of 16 partners and for both spin channels."""

import numpy as np
import pytest

from am1gpu import _abi, workloads as W

pytestmark = pytest.mark.gpu


def _mol(kind, k, seed):
    rng = np.random.default_rng(seed)
    m = W.water_cluster(k, rng) if kind == "water" else W.alkane(k, rng, radical=kind == "radical")
    return (m.numbers, _abi.angstrom_to_bohr(m.xyz), 0.0, m.multiplicity)


def test_split_equals_whole(gpu):
    mols = [_mol(kind, k, 70 + k) for kind, k in (("water", 1), ("water", 2), ("alkane", 16), ("alkane", 17), ("alkane", 18),
                                                  ("radical", 17), ("water", 33), ("water", 34), ("radical", 3))]
    fill = [_mol("water", 20, 200 + i) for i in range(560)]
    assert sum(len(m[0]) for m in mols + fill) >= 32768
    status, whole = gpu.scf_batch(mols + fill)
    assert all(x == 0 for x in status)
    for m, r in zip(mols, whole):
        s = gpu.scf(*m, want_matrices=False)
        assert s["iterations"] == r["iterations"]
        assert s["energy_ev"] == r["energy_ev"] and s["residual"] == r["residual"]
        assert np.array_equal(s["charges"], r["charges"])
