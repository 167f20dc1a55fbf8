"""Return codes of the plain factorisation where no launch can succeed (no GPU)."""
import subprocess
import sys

import pytest

# in a process of its own: other tests count the launches of theirs
PROGRAM = """
import numpy as np
from starpu_gb300.native import load
lib = load()
a, info = np.zeros(4, np.float32), np.zeros(1, np.int32)  # never reached
rc = lib.starpu_gb300_spotrf(None, 5000, a.ctypes.data, 5000, 512, info.ctypes.data)
print(rc, lib.starpu_gb300_launch_count())
"""


def test_nothing_is_enqueued_behind_a_failed_launch(native):
    if native.starpu_gb300_device_count() > 0:
        pytest.skip("needs a machine without a GPU")
    out = subprocess.run([sys.executable, "-c", PROGRAM], capture_output=True, text=True, check=True).stdout
    # GB300_ECUDA; the first diagonal block's launch fails, its panel solve and update are not launched
    assert out.split() == ["-1000", "1"]
