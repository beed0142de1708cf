"""Screen features before and after the host program resets the device (which ends
only its own context): the same values.  In a process of its own, since a
reset ends every other library's state too."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import ctypes as C
import types
import numpy as np
from ps_claude_opt_b200 import native, screen

rng = np.random.default_rng(1)
lens = np.array([40, 60, 50], dtype=np.int32)
obj = types.SimpleNamespace(tim=np.sort(rng.uniform(0, 900, 150)), brightness=1 + 0.2 * rng.standard_normal(150),
                            curve_len=lens, curve_rel=np.ones(3, dtype=np.int32))
freqs = np.linspace(0.02, 0.4, 300)
native.lib()
reset = C.CDLL(next(l.split()[-1] for l in open("/proc/self/maps") if "libcudart.so" in l)).cudaDeviceReset
first = screen.features(obj, freqs)
for _ in range(3):
    assert reset() == 0
    for _ in range(2):
        assert np.array_equal(screen.features(obj, freqs), first)
print("same")
"""


def test_features_after_a_device_reset():
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.strip() == "same"
