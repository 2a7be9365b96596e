"""The marching myMRT step (csrc/fused_march.cuh) in the forms a lattice can take:
every tile candidate of a myMRT lattice, periodic in y (rows wrap around the
box), walls in x, owned and mirrored ranges."""
import numpy as np
import pytest

from multiphaselb_b200 import abi, cases, slabs
from tests.helpers import assert_same, mymrt, run_checker, small_cases, thermal_box
from tests.test_march import MARCH, column

pytestmark = pytest.mark.gpu


def box(nx, ny, periodic):
    """A bubble with noise in T and U; fixedT and bounce-back walls on the axes that
    are not periodic (on one axis at most: their corners would meet)."""
    c = thermal_box(abi.D2Q9, (nx, ny), periodic)
    T0, np_ = c.meta["T"], len(c.patches)
    c.f = dict(c.f, bc_type=[abi.BC_BOUNCEBACK] * np_, bc_value=np.zeros((np_, 3)))
    c.g = mymrt(abi.D2Q9, [abi.BC_FIXEDT] * np_, [(1.02 * T0, 0, 0), (0.98 * T0, 0, 0)][:np_])
    c.eos = dict(c.eos, g=(0.0, -1e-5, 0.0), rho_0=0.0)
    return cases.perturbed(c, du=1e-3)


@pytest.mark.parametrize("nx,ny,periodic", [(2, 2, (True, True)), (3, 9, (True, True)), (28, 33, (True, True)),
                                            (57, 40, (True, True)), (31, 3, (False, True)), (30, 41, (False, True)),
                                            (60, 25, (True, False))])
def test_boxes_match_oracle(gpu_lib, nx, ny, periodic):
    from multiphaselb_b200 import Lattice
    case = box(nx, ny, periodic)
    want = run_checker("port", case, 7)
    with Lattice(case, path=abi.PATH_FUSED, tile_config=MARCH) as lat:
        lat.upload_case()
        lat.initialize()
        lat.step(3)
        lat.step(4)
        assert lat.info()["tile_config"] == MARCH - 1
        assert_same(lat.download(), want, ctx=f"{nx} x {ny} {periodic}")


@pytest.mark.parametrize("make", [lambda: small_cases()["my_column_d2q9"], lambda: column(57, 64, True)])
def test_every_candidate_of_a_mymrt_lattice(gpu_lib, make):
    """All eleven; the tuner times them all and may keep any."""
    from multiphaselb_b200 import Lattice
    case = make()
    want = run_checker("port", case, 4)
    for c in range(12):
        with Lattice(case, path=abi.PATH_FUSED, tile_config=c) as lat:
            lat.upload_case()
            lat.initialize()
            lat.step(4)
            info = lat.info()
            assert c == 0 or info["tile_config"] == c - 1
            if c == 0:
                assert all(t > 0 for t in info["tile_ms"][:11]) and 0 <= info["tile_config"] < 11, info
            assert_same(lat.download(), want, ctx=f"candidate {c - 1}")


@pytest.mark.parametrize("mirror", [False, True])
def test_slabs_as_on_a_tile(gpu_lib, mirror):
    """Slabs stepping on the march against slabs on a tile kernel: with mirrors, the
    march stores owned ranges and the neighbours' halos."""
    case = column(57, 64)
    outs = []
    for tile in (1, MARCH):
        with slabs.FusedSlabRun(case, 3, tile_config=tile, mirror=mirror) as run:
            run.initialize()
            run.step(6)
            outs.append(run.gather())
    assert_same(outs[1], outs[0], fields=[f for f in ("rho", "U", "T", "S", "f", "g") if f in outs[0]], ctx="slabs")
