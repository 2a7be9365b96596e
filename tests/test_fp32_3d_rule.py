"""The FP32 D3Q15 step's choice of its kernel: the rule on the host, and each
kernel at sizes that take it, against the FP64 oracle."""
import os
import shutil
import subprocess
import tempfile

import numpy as np
import pytest

from multiphaselb_b200 import abi, cases
from tests.helpers import run_checker

HERE = os.path.dirname(os.path.abspath(__file__))


def test_rule_on_the_host():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "rule")
        subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a",
                        "-I", os.path.join(HERE, "..", "include"),
                        "-o", exe, os.path.join(HERE, "fp32_3d_rule_check.cu")], check=True, capture_output=True)
        r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("OK"), r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(250, 250, 2), (60, 58, 128), (64, 64, 4), (320, 256, 2), (64, 8, 8), (64, 16, 9),
                                  (192, 192, 8), (128, 128, 64)])
def test_kernels_match_oracle(gpu_lib, dims):
    """The general kernel at four blocks per SM (504 and 480 blocks, partial tiles
    among them) and on flat boxes that the TMA tiles divide, and the TMA-staged
    kernel with either tile; the bounds are those of six FP32 steps at other
    sizes (test_tma_staging.py)."""
    from multiphaselb_b200 import Lattice
    case = cases.perturbed(cases.bubble_case(abi.D3Q15, 8, 2.5, 3.0, 0.75, dims=dims), du=1e-3)
    want = run_checker("port", case, 6)
    with Lattice(case, path=abi.PATH_FUSED, precision=abi.FP32_DEV) as lat:
        lat.upload_case()
        lat.initialize()
        lat.step(4)
        lat.step(2)
        got = lat.download()
    assert np.linalg.norm(got["rho"] - want["rho"]) <= 5e-7 * np.linalg.norm(want["rho"])
    assert np.abs(got["U"] - want["U"]).max() <= 1e-5
