"""Grid reductions (gridred.cuh) end by themselves when a block never arrives: the wait runs out and every
form of the sum gives NaN, on which the Krylov solvers end.  The kernel leaves and the device stays
usable: its second launch sums as it should."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "caffe_old_b200", "csrc")


def test_sums_after_a_lost_wait_are_nan(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "lost_wait")
    cmd = [nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "-DCAFFE_GR_POLLS=2000", "-I", CSRC,
           os.path.join(HERE, "cpp", "lost_wait.cu"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.split("\n")[:2] == ["lost 1 1 1 1", f"whole {64 * 2 * 3} {64 * 2 * 4} {64 * 2 * 1} {64 * 2 * 2}"]
