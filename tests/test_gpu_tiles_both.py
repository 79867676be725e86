"""Odd and even orders in one launch of the tile kernels (k_sp2_step_both, k_commutator_both) against a batch of the
odd ones alone (k_sp2_step8, k_commutator8) and of the even ones alone, bit for bit."""

import numpy as np
import pytest

from am1gpu import _abi, workloads as W

pytestmark = pytest.mark.gpu


def _radical(k, seed):
    m = W.alkane(k, np.random.default_rng(seed), radical=True)
    return (m.numbers, _abi.angstrom_to_bohr(m.xyz), 0.0, m.multiplicity)


def _water(k, seed):
    m = W.water_cluster(k, np.random.default_rng(seed))
    return (m.numbers, _abi.angstrom_to_bohr(m.xyz), 0.0, m.multiplicity)


# orders 6 k + 1, two channels each: enough for a launch per step; and 6 k
ODD = [_radical(k, 70 + k) for k in (21, 21, 22, 23, 31, 32, 42, 64, 76)]
EVEN = [_water(k, 90 + k) for k in (19, 20, 21, 21, 22, 22, 23, 23, 24, 24, 25, 25, 26, 32, 43, 64, 76)]


def test_mixed_equals_alone(gpu):
    parts = []
    for mols in (ODD, EVEN):
        status, res = gpu.scf_batch(mols, want_matrices=True)
        assert all(s == 0 for s in status)
        parts += res
    status, res = gpu.scf_batch(ODD + EVEN, want_matrices=True)
    assert all(s == 0 for s in status)
    for a, b in zip(parts, res):
        assert a["iterations"] == b["iterations"] and a["energy_ev"] == b["energy_ev"]
        assert np.array_equal(a["density"], b["density"])
