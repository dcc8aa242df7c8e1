"""Block -> work layout of the chained 2D passes, checked on the CPU: the check
program (tests/chain_mapping_check.cu) calls the kernel header's own chain_layout
and chain_work over grid shapes, layer widths, block counts and cost factors."""
import os
import shutil
import subprocess

import pytest

from tests.conftest import ROOT


def test_every_row_of_every_stripe_once(tmp_path):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None)
    if nvcc is None:
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "chain_mapping_check")
    cmd = [nvcc, "-std=c++17", "-O2", "-gencode", "arch=compute_103a,code=sm_103a",
           "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "simulation_gb300", "csrc"),
           os.path.join(ROOT, "tests", "chain_mapping_check.cu"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout[-2000:]
