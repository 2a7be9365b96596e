"""The marching D2Q9 step with myMRT heat (csrc/fused_march.cuh): its index
arithmetic on the CPU, and its results against the oracle, bit for bit, at
widths around its 28-column strips, with and without walls in x."""
import os
import shutil
import subprocess
import tempfile

import numpy as np
import pytest

from multiphaselb_b200 import abi, cases
from tests.helpers import assert_same, mymrt, run_checker

HERE = os.path.dirname(os.path.abspath(__file__))
MARCH = 11  # tile_config of the marching candidate


def test_march_indices_in_bounds():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "geom")
        subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a",
                        "-I", os.path.join(HERE, "..", "include"),
                        "-o", exe, os.path.join(HERE, "march_geometry_check.cu")], check=True, capture_output=True)
        r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("OK"), r.stdout + r.stderr


def column(nx, ny, walls_x=False, f_update=1):
    c = cases.column_case(nx, ny, amp=1e-3, width=3.0)
    vals = c.g["bc_value"]
    if walls_x:
        c.nb, c.points, c.patches, c.patch_names = cases.box_mesh(abi.D2Q9, (nx, ny), (False, False))
        c.f = dict(c.f, bc_type=[abi.BC_BOUNCEBACK] * 4, bc_value=np.zeros((4, 3)))
        vals = np.vstack([[vals[0], vals[1]], vals])
    c.g = mymrt(abi.D2Q9, [abi.BC_FIXEDT] * len(c.patches), vals)
    c.f = dict(c.f, update=f_update)
    return cases.perturbed(c, du=1e-3)


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,walls_x,f_update", [(2, 9, False, 1), (27, 12, False, 1), (28, 33, False, 1),
                                                    (29, 12, True, 1), (57, 64, True, 1), (30, 17, False, 0)])
def test_march_matches_oracle(gpu_lib, nx, ny, walls_x, f_update):
    from multiphaselb_b200 import Lattice
    case = column(nx, ny, walls_x, f_update)
    want = run_checker("port", case, 5)
    with Lattice(case, path=abi.PATH_FUSED, tile_config=MARCH) as lat:
        lat.upload_case()
        lat.initialize()
        lat.step(2)
        lat.step(3)
        assert lat.info()["tile_config"] == MARCH - 1
        assert_same(lat.download(), want, ctx=case.name)
