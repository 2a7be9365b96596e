"""Slabs on the fused path with myMRT heat, whose steps reach one plane further
than the others (T of a neighbour holds its heat source), against the
single-domain oracle: the owned planes bit for bit, halos copied or mirrored."""
import pytest

from multiphaselb_b200 import abi, slabs
from tests.helpers import assert_same, run_checker
from tests.test_gpu_march_forms import box
from tests.test_march import MARCH, column

pytestmark = pytest.mark.gpu

CASES = {"column": lambda: column(57, 64), "periodic_y": lambda: box(30, 21, (True, True))}


@pytest.mark.parametrize("tile", [0, 1, MARCH])
@pytest.mark.parametrize("mirror", [False, True])
@pytest.mark.parametrize("name,ranks", [("column", 3), ("periodic_y", 2), ("periodic_y", 5)])
def test_mymrt_slabs_match_oracle(gpu_lib, name, ranks, mirror, tile):
    case = CASES[name]()
    with slabs.FusedSlabRun(case, ranks, mirror=mirror, tile_config=tile) as run:
        assert all(s["lat"].info()["path"] == abi.PATH_FUSED for s in run.slabs)
        run.initialize()
        for steps in (5, 9):
            run.step(steps if steps == 5 else 4)
            assert_same(run.gather(), run_checker("port", case, steps), ctx=f"{name} in {ranks} slabs @{steps}")
