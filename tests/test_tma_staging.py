"""The TMA-staged D3Q15 kernels: their staging (tensor copies, wrapped parts of
face tiles) replayed on the CPU, and the FP32 one against the FP64 oracle."""
import os
import shutil
import subprocess
import tempfile

import numpy as np
import pytest

from multiphaselb_b200 import abi, cases
from tests.helpers import run_checker

HERE = os.path.dirname(os.path.abspath(__file__))


def test_staging_on_the_host():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "geom")
        subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a",
                        "-I", os.path.join(HERE, "..", "include"),
                        "-o", exe, os.path.join(HERE, "fused32_tma_geometry_check.cu")], check=True, capture_output=True)
        r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("OK"), r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(32, 8, 2), (64, 8, 3), (64, 16, 9), (96, 24, 5), (192, 8, 4), (36, 8, 6), (32, 12, 5)])
def test_fp32_3d_steps(gpu_lib, dims):
    """Boxes one or more 64 x 8 and 32 x 8 tiles wide, and two that neither tile
    divides (the general kernel).  Six steps round each population (0.1 at most)
    to FP32 six times: 6 * 6e-8 * 0.1 in a density of 0.3 or a momentum that the
    vapour density 0.016 divides; a wrong neighbour is off by the velocity
    perturbation, 1e-3, at least."""
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


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(16, 8), (24, 20), (96, 64), (256, 256), (300, 290), (512, 530)])
@pytest.mark.parametrize("heat", [False, True])
def test_fp32_2d_steps(gpu_lib, dims, heat):
    """The sizes at which the FP32 2D step changes its kernel (tiles of 32 x 8 up to
    74, 148, 296, 1036 and more), partial tiles among them, in six steps against
    the FP64 oracle; bounds as for the 3D steps (densities 0.02 and more)."""
    from multiphaselb_b200 import Lattice
    if heat:
        case = cases.perturbed(cases.column_case(*dims, amp=1e-3, width=3.0), du=1e-3)
    else:
        case = cases.perturbed(cases.bubble_case(abi.D2Q9, 8, 2.5, 3.0, 0.8, dims=dims), du=1e-3)
    want = run_checker("port", case, 6)
    with Lattice(case, path=abi.PATH_FUSED, precision=abi.FP32_DEV) as lat:
        lat.upload_case()
        lat.initialize()
        lat.step(4)
        lat.step(2)
        got = lat.download()
    for k in ("rho", "T"):
        assert np.linalg.norm(got[k] - want[k]) <= 5e-7 * np.linalg.norm(want[k]), k
    assert np.abs(got["U"] - want["U"]).max() <= 1e-5
