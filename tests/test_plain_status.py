"""Return codes of the plain factorisation where no launch can succeed (no GPU)."""
import numpy as np
import pytest

GB300_ECUDA = -1000


def test_nothing_is_enqueued_behind_a_failed_launch(native):
    if native.starpu_gb300_device_count() > 0:
        pytest.skip("needs a machine without a GPU")
    a, info = np.zeros(4, np.float32), np.zeros(1, np.int32)  # never reached
    before = native.starpu_gb300_launch_count()
    # the first diagonal block's cooperative launch fails; its panel solve and update are not launched
    assert native.starpu_gb300_spotrf(None, 5000, a.ctypes.data, 5000, 512, info.ctypes.data) == GB300_ECUDA
    assert native.starpu_gb300_launch_count() - before == 1
