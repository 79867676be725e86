"""The on-chip tridiagonal reduction at the edges of its column pairs, row groups and cluster sizes (odd and
even orders, the last order a cluster of 1, 2, 4, 8 or 16 CTAs holds and the first of the next)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 7, 8, 15, 16, 17, 31, 32, 33, 63, 64, 65, 66, 127, 128, 129, 130, 164, 165, 166, 167,
                               168, 192, 229, 230, 231, 232, 233, 234, 235, 236, 255, 256, 257, 321, 326, 327, 328, 447, 448, 449,
                               454, 512, 513, 514, 628, 633])
@pytest.mark.parametrize("kind", ["dense", "degenerate", "diagonal"])
def test_eigenvalues(gpu, n, kind):
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n))
    a = 0.5 * (a + a.T)
    if kind == "degenerate":
        q, _ = np.linalg.qr(a)
        a = (q * np.where(np.arange(n) % 3 == 0, -2.0, 1.0)) @ q.T
        a = 0.5 * (a + a.T)
    elif kind == "diagonal":
        a = np.diag(np.diag(a))  # every reflector is zero
    w = gpu.eigvalsh(a)
    # backward stable on both sides: n eps ||A|| each, a factor 5 for the constants
    assert np.max(np.abs(w - np.linalg.eigvalsh(a))) <= 10 * n * 2.2e-16 * max(np.linalg.norm(a, 2), 1e-300)
