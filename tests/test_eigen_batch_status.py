"""Codes of a batch of eigenproblems: every entry is written, also where there is no device to solve the rest."""

import ctypes

import numpy as np

from am1gpu import _abi


def test_every_status_is_written():
    lib = _abi.lib()
    dp = ctypes.POINTER(ctypes.c_double)
    good, bad, big = np.eye(4), np.full((3, 3), np.nan), np.full((500, 500), np.inf)
    mats = [good, bad, None, big, good]
    n = (ctypes.c_int32 * 6)(4, 3, 4, 500, 4, 0)
    a = (dp * 6)(*[None if m is None else m.ctypes.data_as(dp) for m in mats], None)
    ws, vs = [np.zeros(500) for _ in range(6)], [np.zeros((500, 500)) for _ in range(6)]
    w = (dp * 6)(*[x.ctypes.data_as(dp) for x in ws])
    v = (dp * 6)(*[x.ctypes.data_as(dp) for x in vs])
    status = (ctypes.c_int32 * 6)(*[99] * 6)
    rc = lib.am1gpu_symmetric_eigen_batch(6, n, a, w, v, status)
    assert list(status) == [_abi.OK, _abi.LINALG, _abi.INVALID_INPUT, _abi.LINALG, _abi.OK, _abi.OK]
    assert rc == (_abi.LINALG if ws[0][0] == 1.0 else _abi.DEVICE_ERROR)  # solved, or no device here
