"""The network runs after a device reset in the same process: what a launch
needs set on the device is set by the call, not remembered from an earlier one
(the same would fail on a second GPU)."""
import os
import subprocess
import sys

import pytest

from conftest import REPO

pytestmark = pytest.mark.gpu

CODE = """
import ctypes, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
import vnm_gb300
X = np.random.default_rng(1).random((300, 32), dtype=np.float32)
def forward():
    with vnm_gb300.Context(0) as ctx:
        return vnm_gb300.Mlp(ctx, 5).forward(X)
first = forward()
rt = [l.split()[-1] for l in open("/proc/self/maps") if "libcudart.so" in l]
assert ctypes.CDLL(rt[0]).cudaDeviceReset() == 0
assert np.array_equal(forward(), first)
print("ok")
"""


def test_forward_after_a_device_reset():
    out = subprocess.run([sys.executable, "-c", CODE, os.path.join(REPO, "vnm-graph-reordering_gb300")],
                         capture_output=True, text=True, timeout=120)
    assert out.stdout.strip() == "ok", out.stdout + out.stderr[-2000:]
