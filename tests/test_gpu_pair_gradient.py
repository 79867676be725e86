"""The pair forces by a thread per pair (batches of many pairs) against four warps to 32 pairs (few): molecules
alone and in one batch of more pairs than the split takes, at the edges of the pair kinds and of a warp."""

import numpy as np
import pytest

from am1gpu import _abi, workloads as W

pytestmark = pytest.mark.gpu


def _w(k, seed):
    m = W.water_cluster(k, np.random.default_rng(seed))
    return (m.numbers, _abi.angstrom_to_bohr(m.xyz), 0.0, m.multiplicity)


def _a(k, seed, radical=False):
    m = W.alkane(k, np.random.default_rng(seed), radical=radical)
    return (m.numbers, _abi.angstrom_to_bohr(m.xyz), 0.0, m.multiplicity)


def _z(z, x, mult=1):
    return (np.array(z, dtype=np.int32), np.array(x, dtype=np.float64), 0.0, mult)


MOLS = {
    "one atom": (np.array([9], dtype=np.int32), np.zeros((1, 3)), -1.0, 1),
    "two hydrogens": _z([1, 1], [[0, 0, 0], [0.3, 0.2, 1.3]]),
    "one heavy pair": _z([7, 7], [[0, 0, 0], [0.5, 0.1, 2.0]]),
    "one mixed pair": _z([1, 9], [[0, 0, 0], [0.2, 0.3, 1.7]]),
    "third row": _z([16, 17, 1], [[0, 0, 0], [0.3, 0.2, 3.8], [2.4, 0.1, -0.4]]),
    "water": _w(1, 1), "radical": _a(4, 2, True), "11 waters": _w(11, 3), "32 waters": _w(32, 4), "C11H24": _a(11, 5),
}


def test_split_and_whole(gpu):
    filler = [_a(12, 10 + i) for i in range(16)]  # 703 pairs each: past the split's 64 per SM
    status, res = gpu.gradient_batch(list(MOLS.values()) + filler)
    assert all(s == 0 for s in status)
    for (name, mol), r in zip(MOLS.items(), res):
        alone = gpu.scf_gradient(*mol)
        # a component sums at most 95 pairs of 11 parts, each of 100 eV/Bohr at most and rounded to some
        # ten eps: 95 * 11 * 100 * 10 * 2.2e-16
        assert np.max(np.abs(alone["gradient"] - r["gradient"])) < 2.4e-10, name
        assert np.max(np.abs(np.sum(alone["gradient"], axis=0))) < 2.4e-10, name  # +f and -f of every pair
