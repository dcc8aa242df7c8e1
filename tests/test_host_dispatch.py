"""What the 2D entry points launch, checked on the CPU: the check program
(tests/host_dispatch_check.cu) includes their sources with the CUDA runtime and
the kernel launchers replaced by fakes that record their arguments."""
import os
import shutil
import subprocess

import pytest

from tests.conftest import ROOT


@pytest.mark.parametrize("part", ["STEP_N", "ADJOINT"])
def test_launches_and_status_words(tmp_path, part):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None)
    if nvcc is None:
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "host_dispatch_check")
    cmd = [nvcc, "-std=c++17", "-O1", "--expt-relaxed-constexpr", f"-D{part}", "-gencode", "arch=compute_103a,code=sm_103a",
           "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "simulation_gb300", "csrc"),
           os.path.join(ROOT, "tests", "host_dispatch_check.cu"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout[-2000:]
