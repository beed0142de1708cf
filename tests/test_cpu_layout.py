"""Every shared-memory layout that the entry points choose leaves room for the
static shared memory of each kernel that may run it (the teams' kernel holds
the object and the layout, the batch's the current object): a walk over all
object sizes they accept, with the kernels' own layout function."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_chosen_layouts_fit_every_kernel(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not installed")
    exe = str(tmp_path / "layout_driver")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I" + os.path.join(ROOT, "include"), "-I" + os.path.join(ROOT, "ps_claude_opt_b200", "csrc"),
                    "-o", exe, os.path.join(ROOT, "tests", "layout_driver.cu")], check=True, timeout=300)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=300).stdout.split("\n")
    assert out[:-2] == []
    assert int(out[-2]) > 10_000_000
