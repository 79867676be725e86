"""G(P) calls at the ends of their range: no orbitals at all (refused, as a launch without blocks is), one density."""

import numpy as np
import pytest

from am1gpu import _abi, native

pytestmark = pytest.mark.gpu


def test_a_molecule_without_atoms_is_refused(gpu):
    for nrhs in (1, 3):
        with pytest.raises(native.Am1GpuError) as e:
            gpu.g_matrix_batch(np.zeros(0, np.int32), np.zeros((0, 3)), np.zeros((nrhs, 0, 0)))
        assert e.value.code == _abi.DEVICE_ERROR
    # and the library still answers
    assert gpu.scf(np.array([1, 1], np.int32), np.array([[0.0, 0.0, 0.0], [0.0, 0.0, 1.4]]))["status"] == 0
