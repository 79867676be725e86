"""A thread's captured loop serves the next solve only where its kernels' arguments are the same: molecules of
one layout with other coordinates, layouts in turn, and other options, against the same solves in fresh threads."""

import threading

import numpy as np
import pytest

from am1gpu import _abi, workloads as W

pytestmark = pytest.mark.gpu


def _water(k, seed):
    m = W.water_cluster(k, np.random.default_rng(seed))
    return (m.numbers, _abi.angstrom_to_bohr(m.xyz), 0.0, m.multiplicity)


def _alkane(k, seed, radical=False, charge=0.0):
    m = W.alkane(k, np.random.default_rng(seed), radical=radical)
    return (m.numbers, _abi.angstrom_to_bohr(m.xyz), charge, m.multiplicity)


def _fresh(gpu, mol, kw):
    out = {}

    def run():
        out["r"] = gpu.scf(*mol, **kw)

    t = threading.Thread(target=run)
    t.start()
    t.join()
    return out["r"]


SEQUENCES = {
    "one layout": [(_water(4, s), {}) for s in (1, 2, 3)],
    "layouts in turn": [(_water(4, 1), {}), (_alkane(7, 2), {}), (_water(4, 3), {}), (_water(21, 4), {}), (_water(4, 5), {})],
    "other options": [(_water(4, 1), {}), (_water(4, 1), {"max_scf": 3}), (_water(4, 1), {}), (_water(4, 1), {"method": "rm1"}),
                      (_water(4, 1), {"use_diis": False}), (_water(4, 1), {})],
    "spin and charge": [(_alkane(5, 1), {}), (_alkane(5, 1, radical=True), {}), (_alkane(5, 1, charge=2.0), {}), (_alkane(5, 2), {})],
}


@pytest.mark.parametrize("name", list(SEQUENCES))
def test_repeated_solves_equal_fresh_ones(gpu, name):
    for mol, kw in SEQUENCES[name]:
        here, fresh = gpu.scf(*mol, **kw), _fresh(gpu, mol, kw)
        assert here["status"] == fresh["status"] and here["iterations"] == fresh["iterations"]
        assert here["energy_ev"] == fresh["energy_ev"]  # the same kernels in the same order: the same bits
        assert np.array_equal(here["density"], fresh["density"])
