"""A thread's priority holds for every stream its calls run on, also where they exist already: beside a kernel that fills the
GPU for a long time, calls of a higher priority do not wait for it to end."""

import threading
import time

import numpy as np
import pytest

from am1gpu import _abi, workloads as W

pytestmark = pytest.mark.gpu


def _background():
    """A launcher of one long kernel of many short blocks, and its duration in seconds."""
    import torch

    d = 64
    while True:
        x = torch.rand(6000, d, dtype=torch.float64, device="cuda")
        torch.cdist(x, x, p=3.5)  # a block per pair of rows
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        torch.cdist(x, x, p=3.5)
        b.record()
        torch.cuda.synchronize()
        ms = a.elapsed_time(b)
        if ms > 150.0 or d >= 4096:
            return (lambda: torch.cdist(x, x, p=3.5)), 1e-3 * ms
        d *= 2


def test_streams_that_exist_follow_the_priority(gpu):
    import torch

    launch, long = _background()
    if long < 0.1:
        pytest.skip("no kernel long enough to wait for")
    rng = np.random.default_rng(1)
    mats = [(lambda a: a + a.T)(rng.standard_normal((64, 64))) for _ in range(8)]  # on the device, a stream a group
    m = W.water_cluster(20, rng)
    xyz = _abi.angstrom_to_bohr(m.xyz)
    dens = rng.standard_normal((60, 120, 120))
    dens = dens + dens.transpose(0, 2, 1)  # several pipelines
    calls = {"eigh_batch": lambda: gpu.eigh_batch(mats), "g_matrix_batch": lambda: gpu.g_matrix_batch(m.numbers, xyz, dens),
             "scf": lambda: gpu.scf(m.numbers, xyz)}
    took = {}

    def work():
        for f in calls.values():  # every stream exists, at priority 0
            f()
        gpu.set_stream_priority(-5)
        for name, f in calls.items():
            f()
            torch.cuda.synchronize()
            launch()
            time.sleep(0.01)
            t = time.perf_counter()
            f()
            took[name] = time.perf_counter() - t
            torch.cuda.synchronize()

    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert set(took) == set(calls)
    assert all(x < 0.5 * long for x in took.values()), (took, long)
