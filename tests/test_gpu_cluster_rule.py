"""Which channels above 112 orbitals purify in a cluster each depends on how many the batch has and how large they are:
at the lines of that rule a molecule's result is its own, bit for bit, and a batch is not slower than a larger one."""

import numpy as np
import pytest

from am1gpu import _abi, native, workloads as W

pytestmark = pytest.mark.gpu


def _waters(k, seed):
    m = W.water_cluster(k, np.random.default_rng(seed))
    return (m.numbers, _abi.angstrom_to_bohr(m.xyz), 0.0, m.multiplicity)


@pytest.mark.parametrize("sizes", [[32] * 7, [32] * 8, [33] * 15, [32] * 16, [33] * 17, [64] * 8, [48] * 9,
                                   [70] + [33] * 9 + [32] * 6, [70, 64, 55, 53, 43, 41] + [20] * 5, [76, 70, 32, 19, 18, 3]])
def test_results_are_a_molecules_own(gpu, sizes):
    mols = [_waters(k, 7 + i) for i, k in enumerate(sizes)]
    status, res = gpu.scf_batch(mols)
    assert not any(status) and gpu.last_call_stats()["eigen_fallbacks"] == 0
    for i in {0, len(sizes) // 2, len(sizes) - 1}:
        alone = gpu.scf(*mols[i], want_matrices=False)
        assert res[i]["energy_ev"] == alone["energy_ev"] and res[i]["iterations"] == alone["iterations"]


def _device_ms(count, size):
    b = native.Batch([_waters(size, i) for i in range(count)])
    ms = []
    for _ in range(5):
        assert b.run() == 0
        ms.append(native.last_call_stats()["device_ms"])
    return min(ms)


@pytest.mark.parametrize("count,size", [(8, 74), (16, 64), (16, 74)])
def test_clusters_only_where_they_are_faster(gpu, count, size):
    # 17 channels take the launch-per-step tiles; fewer of the same size cannot take longer (10% for the clocks)
    assert _device_ms(count, size) < 1.1 * _device_ms(17, size)
