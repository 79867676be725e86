"""Purifications at the edge of the cluster kernel (448 orbitals): the orders just past it, which the cluster Jacobi
still takes, purify as well, without a fall-back to the eigensolver, alone as in a batch."""

import numpy as np
import pytest

from am1gpu import _abi, workloads as W

pytestmark = pytest.mark.gpu


def _mol(kind, size):
    rng = np.random.default_rng(size)
    m = W.water_cluster(size, rng) if kind == "water" else W.alkane(size, rng, radical=kind == "radical")
    return (m.numbers, _abi.angstrom_to_bohr(m.xyz), 0.0, m.multiplicity)


@pytest.mark.parametrize("kind,size,nao", [("alkane", 74, 446), ("water", 75, 450), ("radical", 75, 451), ("alkane", 75, 452),
                                           ("water", 76, 456)])
def test_purifies_past_the_cluster_kernel(gpu, kind, size, nao):
    mol = _mol(kind, size)
    r = gpu.scf(*mol, want_matrices=False)
    stats = gpu.last_call_stats()
    assert r["status"] == 0 and r["nao"] == nao
    assert stats["eigen_fallbacks"] == 0, stats
    # 17 channels more: none of them purifies in a cluster; the bits of a molecule are its own
    status, res = gpu.scf_batch([mol] + [_mol("water", 32)] * 17)
    assert not any(status) and gpu.last_call_stats()["eigen_fallbacks"] == 0
    assert res[0]["energy_ev"] == r["energy_ev"] and res[0]["iterations"] == r["iterations"]
