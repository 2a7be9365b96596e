"""Surface-tension lattices on every tile candidate of the fused path and on the
table kernels, isothermal and with heat (liTempMRT, myMRT), bit for bit against
the oracle; and a forced candidate runs the kernel of its own tile."""
import pytest

from multiphaselb_b200 import abi, cases
from tests.captured import captured_kernels
from tests.helpers import (assert_same, cylinder_d2q9, mymrt, run_checker, surface_tension_d2q9, surface_tension_d3q15)

pytestmark = pytest.mark.gpu

# tile_config -> tile of the candidate (csrc/fused.cuh, CFG2 and CFG3; the march
# and the table kernels have none)
TILES2 = {1: (32, 8), 2: (32, 4), 3: (64, 4), 4: (16, 8), 5: (64, 4), 6: (16, 8), 7: (32, 8), 8: (32, 4), 9: (32, 8),
          10: (16, 8), 11: None}
TILES3 = {1: (32, 8), 2: (32, 8), 3: (32, 4), 4: (64, 4), 5: (32, 16), 6: None, 7: (32, 4), 8: (32, 8), 9: (32, 16),
          10: (64, 8)}


def st(c):
    c.f = dict(c.f, surface_tension=1, kappa_st=0.4)
    return c


def column(my=False):
    """41 x 30, more than one tile of every shape, partial ones among them."""
    c = cases.column_case(41, 30, amp=1e-3, width=3.0)
    if my:
        c.g = mymrt(abi.D2Q9, [abi.BC_FIXEDT] * 2, c.g["bc_value"])
    return cases.perturbed(st(c), du=1e-3)


def cylinder(my=False):
    c = cylinder_d2q9()
    if my:
        c.g = mymrt(abi.D2Q9, c.g["bc_type"], c.g["bc_value"])
    return st(c)


CASES = {"column": column, "my_column": lambda: column(True), "bubble_walls": surface_tension_d2q9,
         "walls3d": surface_tension_d3q15,
         "bubble3d": lambda: cases.perturbed(st(cases.bubble_case(abi.D3Q15, 8, 2.5, 3.0, 0.75, dims=(64, 16, 5))), du=1e-3)}


@pytest.mark.parametrize("name", list(CASES))
def test_every_candidate(gpu_lib, name):
    import torch
    from multiphaselb_b200 import Lattice, MplbError
    case = CASES[name]()
    want = run_checker("port", case, 5)
    tiles = TILES2 if case.lattice == abi.D2Q9 else TILES3
    ran = []
    for c, tile in tiles.items():
        stream = torch.cuda.Stream()
        with Lattice(case, path=abi.PATH_FUSED, tile_config=c, stream=stream.cuda_stream) as lat:
            lat.upload_case()
            lat.initialize()
            try:
                lat.step(1)
            except MplbError as e:
                assert "does not take this lattice" in str(e), e
                continue
            lat.step(4)
            assert lat.info()["tile_config"] == c - 1
            assert_same(lat.download(), want, ctx=f"{name} candidate {c - 1}")
            lat.step(1)
            lat.sync()
            kernels = captured_kernels(stream, lambda: lat.step(2))
        if tile:
            assert any(args[:2] == tile for _, args in kernels), (c, kernels)
        else:
            assert [k for k, _ in kernels] == ["k_table_sum", "k_table_finish"] * 2, kernels
        ran.append(c)
    # the march has no surface tension; TMA tiles take the periodic box, which they all divide
    assert ran == list(range(1, (6 if name == "walls3d" else 10) + 1)), ran
    with Lattice(case, path=abi.PATH_FUSED) as lat:
        lat.upload_case()
        lat.initialize()
        lat.step(5)
        assert lat.info()["tile_config"] + 1 in ran
        assert_same(lat.download(), want, ctx=f"{name} autotuned")


@pytest.mark.parametrize("name", ["cylinder", "my_cylinder", "column", "my_column", "walls3d"])
def test_table_kernels(gpu_lib, name):
    from multiphaselb_b200 import Lattice
    case = {"cylinder": cylinder, "my_cylinder": lambda: cylinder(True)}.get(name, CASES.get(name))()
    with Lattice(case, path=abi.PATH_OPERATORS) as lat:
        lat.upload_case()
        lat.initialize()
        done = 0
        for chunk in (1, 4):
            lat.step(chunk)
            done += chunk
            assert_same(lat.download(), run_checker("port", case, done), ctx=f"{name} after {done}")
        before = lat.info()["kernel_launches"]
        lat.step(1)
        lat.step(9)
        assert lat.info()["kernel_launches"] - before <= 2 + 3 * 10  # two collisions to enter, two or three a step
