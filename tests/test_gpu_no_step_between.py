"""Calls that bring a lattice of the fused path into its stepping state without a
step (monitor, copy_state, a batch run of no steps) leave the reference state to be
read, and the steps after them, as they were."""
import numpy as np
import pytest

from multiphaselb_b200 import abi
from tests.helpers import small_cases

pytestmark = pytest.mark.gpu


def same(a, b):
    for k in a:
        assert np.array_equal(a[k], b[k]), k


def states(lat, steps, call):
    """The state after `steps` steps and `call`, and two steps later."""
    lat.upload_case()
    lat.initialize()
    if steps:
        lat.step(steps)
        lat.download()
    call(lat)
    first = lat.download()
    call(lat)
    lat.step(2)
    return first, lat.download()


@pytest.mark.parametrize("steps", [0, 3])
@pytest.mark.parametrize("precision", [abi.FP64, abi.FP32_DEV])
@pytest.mark.parametrize("name", ["bubble_d2q9", "column_d2q9", "bubble_d3q15", "walls_d3q15"])
def test_monitor(gpu_lib, name, precision, steps):
    from multiphaselb_b200 import Lattice
    got = []
    for call in (lambda lat: None, lambda lat: lat.monitor()):
        with Lattice(small_cases()[name], path=abi.PATH_FUSED, precision=precision) as lat:
            got.append(states(lat, steps, call))
    same(got[0][0], got[1][0])
    same(got[0][1], got[1][1])


def test_copy_state(gpu_lib):
    from multiphaselb_b200 import Lattice
    case = small_cases()["my_column_d2q9"]
    with Lattice(case, path=abi.PATH_FUSED) as a, Lattice(case, path=abi.PATH_FUSED) as b:
        for lat in (a, b):
            lat.upload_case()
            lat.initialize()
        want = b.download()
        a.copy_state(b, 0, 0, case.n)
        same(want, b.download())


def test_batch_without_steps(gpu_lib):
    from multiphaselb_b200 import Batch, Lattice
    case = small_cases()["bubble_d2q9"]
    lats = [Lattice(case, path=abi.PATH_FUSED, precision=abi.FP32_DEV) for _ in range(2)]
    for lat in lats:
        lat.upload_case()
        lat.initialize()
    want = lats[0].download()
    with Batch(lats, check_interval=2) as batch:
        batch.run(0)
        same(want, lats[0].download())
        batch.filter([0, 0])
        batch.average()
        same(want, lats[1].download())
    for lat in lats:
        lat.close()


def test_monitor_before_a_replay(gpu_lib):
    """The steps of a caller's graph run without the handle's knowledge: what they
    leave is read, not the state before the monitor."""
    import torch
    from multiphaselb_b200 import Lattice
    case = small_cases()["column_d2q9"]
    with Lattice(case, path=abi.PATH_FUSED) as lat:
        lat.upload_case()
        lat.initialize()
        lat.step(2)
        lat.download()
        lat.step(4)
        want = lat.download()
    s = torch.cuda.Stream()
    with Lattice(case, path=abi.PATH_FUSED, stream=s.cuda_stream) as lat:
        lat.upload_case()
        lat.initialize()
        lat.step(2)
        graph = torch.cuda.CUDAGraph()
        lat.sync()
        with torch.cuda.graph(graph, stream=s):
            lat.step(2)
        lat.download()
        lat.monitor()
        with torch.cuda.stream(s):
            graph.replay()
        lat.monitor()
        with torch.cuda.stream(s):
            graph.replay()
        torch.cuda.synchronize()
        same(want, lat.download())
        del graph
