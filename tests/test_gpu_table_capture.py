"""A step of a lattice on the operator path while another stream of the program
is being captured: the steps are no part of the capture, whichever handle takes
them and whether or not it is its first step."""
import pytest

from multiphaselb_b200 import abi
from tests.helpers import assert_same, run_checker, small_cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("own_stream", [True, False])
@pytest.mark.parametrize("name", ["cylinder_d2q9", "bubble_d2q9"])
def test_first_step_during_another_capture(gpu_lib, name, own_stream):
    import torch

    from multiphaselb_b200 import Lattice
    case = small_cases()[name]
    mine = None if own_stream else torch.cuda.Stream()
    x = torch.zeros(64, device="cuda")
    torch.cuda.synchronize()
    with Lattice(case, path=abi.PATH_OPERATORS, stream=None if own_stream else mine.cuda_stream) as lat:
        lat.upload_case()
        lat.initialize()
        lat.sync()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):  # global capture mode
            x.add_(1.0)
            lat.step(2)
            x.add_(1.0)
        lat.step(3)
        graph.replay()
        torch.cuda.synchronize()
        assert float(x[0]) == 2.0
        assert_same(lat.download(), run_checker("port", case, 5), ctx=name)
        del graph
