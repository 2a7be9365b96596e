"""CPU check of the way out of the TMA-staged D3Q15 kernels after a wait that ran
out: no thread leaves while its copies into shared memory are in flight."""
import os
import shutil
import subprocess
import tempfile

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_no_copy_in_flight_when_a_thread_leaves():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "leave")
        subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "--extended-lambda",
                        "-gencode", "arch=compute_100a,code=sm_100a",
                        "-o", exe, os.path.join(HERE, "tma_leave_check.cu")], check=True, capture_output=True)
        r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("OK"), r.stdout + r.stderr
