"""A solve that forms no F* (no iteration allowed, or an energy that is not finite in the first) reports the spectrum of a
zero matrix, not one that another solve left in the same memory."""

import numpy as np
import pytest

from am1gpu import _abi, native, workloads as W

pytestmark = pytest.mark.gpu


def _mol(kind, size):
    rng = np.random.default_rng(size)
    m = W.water_cluster(size, rng) if kind == "water" else W.alkane(size, rng, radical=kind == "radical")
    return m.numbers, _abi.angstrom_to_bohr(m.xyz), 0.0, m.multiplicity


@pytest.mark.parametrize("kind,size", [("water", 1), ("radical", 4), ("water", 20), ("water", 80)])
def test_spectrum_without_an_iteration(gpu, kind, size):
    z, xyz, q, mult = _mol(kind, size)
    assert gpu.scf(z, xyz, q, mult)["status"] == 0  # leaves its F* in the workspace
    none = gpu.scf(z, xyz, q, mult, max_scf=0, want_matrices=False)
    assert none["status"] == 3 and none["iterations"] == 0
    together = np.zeros_like(xyz)  # every atom on the first
    lost = gpu.scf(z, together, q, mult, want_matrices=False)
    assert lost["status"] in (3, 4, 5)
    for r in [none] + ([lost] if lost["iterations"] <= 1 and lost["status"] == 4 else []):
        for e in [r["mo_energies"], [r["homo_ev"], r["lumo_ev"]]] + ([r["beta_energies"]] if r["unrestricted"] else []):
            assert np.all(np.abs(e) < 1e-250), e


def test_a_resident_batch_run_again(gpu):
    good, bad = _mol("water", 2), _mol("water", 3)
    bad = (bad[0], np.zeros_like(bad[1]), 0.0, 1)
    first = native.scf_batch([good, bad])[1][1]
    rb = native.ResidentBatch([good, bad])
    try:
        for _ in range(2):
            rb.run()
            status, res = rb.results()
            assert status[0] == 0 and status[1] != 0
            assert np.array_equal(res[1]["mo_energies"], first["mo_energies"])
    finally:
        rb.close()
