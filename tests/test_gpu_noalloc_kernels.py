"""The allocation-free entry point runs single CTAs or teams of them, whichever suits
the number of fits, and the first call with work sets up both kernels: later
calls with any number of fits leave the free device memory as it is.  In a
process of its own, where no other test has loaded a kernel."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import dataclasses
import sys
sys.path.insert(0, "tests")
import numpy as np
import torch
from conftest import prepared
from ps_claude_opt_b200 import native

torch.zeros(1, device="cuda")
native.reserve_noalloc(0)
for kind in ("mixed", "lmax8"):
    obj = dataclasses.replace(prepared(kind), stop_condition=2.0)
    for i, n in enumerate((FIRST, 1, 10, 30, 70, 148, 200)):
        native.fit_items_noalloc(obj, np.ones(n, dtype=np.int32), np.arange(n, dtype=np.int32) % 10)
        free = torch.cuda.mem_get_info()[0]
        if i == 0:
            first = free
        assert free == first, (kind, n, free, first)
print("same")
"""


@pytest.mark.parametrize("first", [300, 1])
def test_later_calls_load_nothing(first):
    r = subprocess.run([sys.executable, "-c", PROGRAM.replace("FIRST", str(first))], cwd=ROOT, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.strip() == "same"
