"""Small calls prepare their matrices on the host, larger ones on the device: a matrix's eigenvalues and vectors are
the same bits either way, and non-finite input is refused by both."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sym(n, seed):
    a = np.random.default_rng(seed).standard_normal((n, n))
    a = a + a.T
    a[np.triu_indices(n, 1)] += 1.0  # only the lower triangle counts
    return a


@pytest.mark.parametrize("n", [1, 2, 3, 31, 32, 33, 64, 65, 97, 126, 127])
def test_small_and_large_calls_agree(gpu, n):
    a = _sym(n, n)
    w, v = gpu.eigh(a)  # n^2 of 16000 elements: 126 rows on the host, 127 on the device
    fill = [_sym(60, k) for k in range(5)]
    status, pairs = gpu.eigh_batch([a] + fill)  # 18000 elements more: the device
    assert not any(status)
    assert np.array_equal(pairs[0][0], w) and np.array_equal(pairs[0][1], v)
    ref = np.linalg.eigvalsh(a, UPLO="L")
    assert np.max(np.abs(w - ref)) < 6 * n * 2.2e-16 * 4 * n * np.max(np.abs(a))


@pytest.mark.parametrize("fill", [0, 5])
def test_non_finite_in_either_triangle(gpu, fill):
    good, low, up = _sym(7, 1), _sym(6, 2), _sym(6, 3)
    low[5, 0], up[0, 5] = np.nan, np.inf
    status, pairs = gpu.eigh_batch([good, low, up] + [_sym(60, k) for k in range(fill)])
    assert status == [0, 5, 5] + [0] * fill
    assert np.array_equal(pairs[0][0], gpu.eigh(good)[0])

