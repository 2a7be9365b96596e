"""Steps of the operator path in fused kernels on the neighbour table
(csrc/fused_table.cuh), bit for bit against the oracle: steps in chunks with
downloads, operator calls and the equilibrium monitor between them, and
lattices whose boundaries keep the operators."""
import numpy as np
import pytest

from multiphaselb_b200 import abi
from oracle import oracle as orc
from tests.helpers import assert_same, small_cases

pytestmark = pytest.mark.gpu

FUSED = ["cylinder_d2q9", "column_d2q9", "bubble_d2q9", "st_d2q9", "my_column_d2q9", "walls_d3q15", "st_d3q15",
         "my_slab_d3q15"]
# the last one's walls meet: its fixedT nodes read what another patch writes
OPERATORS = ["lid_d2q9", "outflow_d2q9", "outflow_d3q15", "outflow_corner_d2q9", "my_walls_d3q15"]


@pytest.mark.parametrize("name", FUSED + OPERATORS)
def test_chunks_and_operators_between(gpu_lib, name):
    from multiphaselb_b200 import Lattice
    case = small_cases()[name]
    k = orc.Checker("port", case)
    k.upload_case()
    k.initialize()
    with Lattice(case, path=abi.PATH_OPERATORS) as lat:
        lat.upload_case()
        lat.initialize()
        for chunk in (1, 4, 3):
            k.step(chunk)
            lat.step(chunk)
            assert_same(lat.download(), k.download(), ctx=f"{name} after chunk {chunk}")
        k.op(orc.OP_COLLISION, abi.FIELD_F)
        lat.collision(abi.FIELD_F)
        k.op(orc.OP_LBSTREAM, abi.FIELD_F)
        lat.lbstream(abi.FIELD_F)
        k.step(2)
        lat.step(2)
        lat.monitor(reset=True)
        k.step(2)
        lat.step(2)
        drho, mass = lat.monitor()
        got = lat.download()
        assert_same(got, k.download(), ctx=f"{name} after operators")
        assert np.isfinite(drho) and abs(mass - got["rho"].sum()) <= 1e-12 * mass


@pytest.mark.parametrize("name,fused", [(n, True) for n in FUSED] + [(n, False) for n in OPERATORS])
def test_launches_per_step(gpu_lib, name, fused):
    """Two or three kernels a step where the fused kernels take the lattice."""
    from multiphaselb_b200 import Lattice
    case = small_cases()[name]
    with Lattice(case, path=abi.PATH_OPERATORS) as lat:
        lat.upload_case()
        lat.initialize()
        lat.step(1)
        before = lat.info()["kernel_launches"]
        lat.step(10)
        per_step = (lat.info()["kernel_launches"] - before) / 10
        assert per_step <= 3 if fused else per_step > 3, per_step


@pytest.mark.parametrize("name", ["walls_d3q15", "st_d3q15", "bubble_d3q15"])
def test_table_candidate(gpu_lib, name):
    """The neighbour-table kernels as a candidate of the fused D3Q15 path."""
    from multiphaselb_b200 import Lattice
    case = small_cases()[name]
    k = orc.Checker("port", case)
    k.upload_case()
    k.initialize()
    with Lattice(case, path=abi.PATH_FUSED, tile_config=6) as lat:
        lat.upload_case()
        lat.initialize()
        for chunk in (1, 6):
            k.step(chunk)
            lat.step(chunk)
            assert_same(lat.download(), k.download(), ctx=f"{name} after {chunk}")
        assert lat.info()["tile_config"] == 5


@pytest.mark.parametrize("warmup", [0, 3])
@pytest.mark.parametrize("name", ["cylinder_d2q9", "my_column_d2q9", "bubble_d2q9"])
def test_captured_steps(gpu_lib, name, warmup):
    """Steps captured on the caller's stream replay as the operators do: from
    the state the handle holds then, also after downloads and other steps."""
    import torch

    from multiphaselb_b200 import Lattice
    case = small_cases()[name]
    k = orc.Checker("port", case)
    k.upload_case()
    k.initialize()
    stream = torch.cuda.Stream()
    with Lattice(case, path=abi.PATH_OPERATORS, stream=stream.cuda_stream) as lat:
        lat.upload_case()
        lat.initialize()
        if warmup:
            lat.step(warmup)
            k.step(warmup)
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            lat.step(2)
        for replays in (1, 2):
            for _ in range(replays):
                with torch.cuda.stream(stream):
                    graph.replay()
                k.step(2)
            assert_same(lat.download(), k.download(), ctx=f"{name} after {replays} replays")
            lat.step(2)
            k.step(2)
        del graph
