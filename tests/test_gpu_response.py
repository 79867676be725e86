"""am1gpu_g_matrix_batch in chunks and pipelines: every right-hand side's result is that of a call of its
own, bit for bit, at the edges of a chunk and for atoms in an order that the internal one (heavy atoms
first) does not keep; and the result is G(P) = J(P) - K(P/2) of am1gpu_build_fock."""

import numpy as np
import pytest

from am1gpu import _abi, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,nrhs", [(1, 1), (1, 65), (2, 64), (20, 19), (43, 4), (43, 9)])
def test_chunks(gpu, k, nrhs):
    m = W.water_cluster(k, np.random.default_rng(k))
    order = np.random.default_rng(7).permutation(3 * k)
    z, xyz = m.numbers[order], _abi.angstrom_to_bohr(m.xyz)[order]
    n = 6 * k
    d = np.random.default_rng(nrhs).standard_normal((nrhs, n, n)) * 0.1
    d = d + d.transpose(0, 2, 1)
    g = gpu.g_matrix_batch(z, xyz, d)
    h, _ = gpu.build_core(z, xyz)
    for r in sorted({0, nrhs // 2, nrhs - 1}):
        assert np.array_equal(g[r], gpu.g_matrix_batch(z, xyz, d[r][None])[0]), r
        # the same sums but for H_core: H of up to a few thousand eV added and taken off again costs its rounding
        f = gpu.build_fock(z, xyz, d[r], d[r], 0.5)
        assert np.max(np.abs(f - h - g[r])) < 8 * 2.2e-16 * max(np.max(np.abs(f)), np.max(np.abs(h)))
