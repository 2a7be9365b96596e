"""Device memory of the neighbour-table candidate of the fused D3Q15 path: its
scratch, 8 bytes a node, is held only by lattices that step on it."""
import pytest

from multiphaselb_b200 import abi, cases
from tests.helpers import assert_same, run_checker

pytestmark = pytest.mark.gpu

# bytes a node of a D3Q15 lattice with a flow only: table 60, flag 1, rho T S p T2 40,
# U Fi Ft U2 96, two FP64 population buffers 240; FP32 form two more of 60; a program index
# with boundaries; tables of fixed size and patch lists below 1 byte a node at these sizes
BASE, FP32 = 437, 120


def box(dims, walls):
    c = cases.bubble_case(abi.D3Q15, 8, 2.5, 3.0, 0.75, dims=dims)
    if walls:
        c.nb, c.points, c.patches, c.patch_names = cases.box_mesh(abi.D3Q15, c.dims, (True, True, False))
        c.periodic = (True, True, False)
        c.f = dict(c.f, bc_type=[abi.BC_BOUNCEBACK] * 2, bc_value=[[0, 0, 0]] * 2)
    return cases.perturbed(c, du=1e-3)


def per_node(lat, n):
    return lat.info()["device_bytes"] / n


@pytest.mark.parametrize("walls", [False, True])
@pytest.mark.parametrize("precision", [abi.FP64, abi.FP32_DEV])
def test_scratch_only_where_the_candidate_steps(gpu_lib, precision, walls):
    from multiphaselb_b200 import Lattice
    case = box((64, 32, 40), walls)
    n = case.n
    base = BASE + (1 if walls else 0) + (FP32 if precision == abi.FP32_DEV else 0)
    want = run_checker("port", case, 3)
    for tile in (0, 3, 6) if precision == abi.FP64 else (0,):
        with Lattice(case, path=abi.PATH_FUSED, precision=precision, tile_config=tile) as lat:
            created = per_node(lat, n)
            assert base <= created < base + 2, (created, base)
            lat.upload_case()      # staging for vectors: 24
            lat.initialize()
            lat.step(1)
            cfg = lat.info()["tile_config"]
            table = precision == abi.FP64 and cfg == 5
            assert (tile == 0) or cfg == (tile - 1)
            stepped = per_node(lat, n) - created - 24
            assert stepped == (8 if table else 0), (tile, cfg, stepped)
            lat.step(2)
            if precision == abi.FP64:
                assert_same(lat.download(), want, fields=("rho", "U", "f"), ctx=f"tile_config {tile}")


def test_slab_does_not_hold_it(gpu_lib):
    """A lattice whose steps store an owned range only never steps on the
    candidate, tuned or forced."""
    from multiphaselb_b200 import Lattice
    case = box((32, 32, 24), True)
    for tile in (0, 6):
        with Lattice(case, path=abi.PATH_FUSED, tile_config=tile) as lat:
            lat.set_owned(32 * 32, 22 * 32 * 32)
            lat.upload_case()
            lat.initialize()
            created = lat.info()["device_bytes"]
            lat.step(2)
            lat.set_owned(0, 0)
            lat.step(1)
            assert lat.info()["device_bytes"] == created, tile
