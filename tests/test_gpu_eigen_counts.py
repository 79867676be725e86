"""More small matrices in one call than a grid's y and z extents hold."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 5])
def test_seventy_thousand_matrices(gpu, n):
    rng = np.random.default_rng(n)
    a = rng.standard_normal((70000, n, n))
    a = a + a.transpose(0, 2, 1)
    status, pairs = gpu.eigh_batch(list(a))
    assert not any(status)
    ref = np.linalg.eigvalsh(a)
    got = np.array([w for w, _ in pairs])
    # n eps (||A|| + shift) a sweep, half a dozen sweeps, the shift up to the Gershgorin bound n max|a|
    assert np.max(np.abs(got - ref)) < 6 * n * 2.2e-16 * 2 * n * np.max(np.abs(a))
    v = np.array([v for _, v in pairs])
    assert np.max(np.abs(v.transpose(0, 2, 1) @ v - np.eye(n))) < 100 * n * 2.2e-16


def test_device_memory_per_matrix(gpu):
    # three n x n matrices (input, C^T, vectors) and a few vectors each, so that as many fit the device as can
    import threading

    import torch

    n, count = 448, 48
    rng = np.random.default_rng(1)
    mats = []
    for _ in range(count):
        a = rng.standard_normal((n, n))
        mats.append(a + a.T)
    used = {}

    def run():
        gpu.eigh(np.eye(2))  # the thread's streams and the device's own buffers
        free = torch.cuda.mem_get_info()[0]
        status, pairs = gpu.eigh_batch(mats)
        used["bytes"] = free - torch.cuda.mem_get_info()[0]
        used["ok"] = not any(status) and all(np.all(np.diff(w) >= 0.0) for w, _ in pairs)

    t = threading.Thread(target=run)  # a workspace of its own
    t.start()
    t.join()
    assert used["ok"]
    assert used["bytes"] < 3.3 * 8 * n * n * count
