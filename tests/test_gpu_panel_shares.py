"""Host threads that reduce large matrices at the same time share the GPU: each panel then runs on fewer CTAs of more shares
each, and the results are the bits of a lone call."""

import threading

import numpy as np
import pytest

from am1gpu import _abi, workloads as W

pytestmark = pytest.mark.gpu


def _sym(n, seed):
    a = np.random.default_rng(seed).standard_normal((n, n))
    return a + a.T + np.diag(np.linspace(-30.0, 30.0, n))


@pytest.mark.parametrize("threads", [2, 3, 5])
def test_threads_get_a_lone_calls_bits(gpu, threads):
    mats = [_sym(n, n) for n in (700, 777, 1001, 2047, 2050)]
    m = W.water_cluster(120, np.random.default_rng(2))  # 720 orbitals
    xyz = _abi.angstrom_to_bohr(m.xyz)
    lone = [gpu.eigvalsh(a) for a in mats]
    w0, v0 = gpu.eigh(mats[0])
    e0 = gpu.scf(m.numbers, xyz, want_matrices=False)["mo_energies"]
    start, wrong = threading.Barrier(threads), []

    def work(i):
        start.wait()
        for k in range(len(mats)):
            a = (k + i) % len(mats)
            if not np.array_equal(gpu.eigvalsh(mats[a]), lone[a]):
                wrong.append(("eigvalsh", a))
        w, v = gpu.eigh(mats[0])
        if not (np.array_equal(w, w0) and np.array_equal(v, v0)):
            wrong.append("eigh")
        if not np.array_equal(gpu.scf(m.numbers, xyz, want_matrices=False)["mo_energies"], e0):
            wrong.append("scf")

    ts = [threading.Thread(target=work, args=(i,)) for i in range(threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not wrong, wrong


def test_reductions_of_threads_run_side_by_side(gpu):
    import time

    a = _sym(1000, 1)

    def best(threads):
        times = []
        for _ in range(3):
            start, done = threading.Barrier(threads + 1), []

            def work():
                gpu.eigvalsh(a)
                start.wait()
                for _ in range(4):
                    gpu.eigvalsh(a)
                done.append(time.perf_counter())

            ts = [threading.Thread(target=work) for _ in range(threads)]
            for t in ts:
                t.start()
            start.wait()
            t0 = time.perf_counter()
            for t in ts:
                t.join()
            times.append((max(done) - t0) / (4 * threads))
        return min(times)

    # one after the other a call of six threads takes 0.85 of a lone one (the copies overlap), three at a time a third of 1.15
    assert best(6) < 0.6 * best(1)
