"""The buffers of the table kernels on the operator path: one allocation, made at
the first step of a handle, and left without loss."""
import numpy as np
import pytest

from multiphaselb_b200 import abi
from tests.helpers import assert_same, run_checker, small_cases
from tests.test_gpu_memory_limit import Nearly, channel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["cylinder_d2q9", "my_column_d2q9", "bubble_d3q15"])
def test_one_allocation(gpu_lib, name):
    import torch
    from multiphaselb_b200 import Lattice
    case = small_cases()[name]
    with Lattice(case, path=abi.PATH_OPERATORS) as lat:
        lat.upload_case()
        lat.initialize()
        lat.sync()
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU,
                                                torch.profiler.ProfilerActivity.CUDA]) as prof:
            lat.step(3)
            lat.sync()
        calls = [e.name for e in prof.events()]
        assert sum("cudaLaunchKernel" in c for c in calls) >= 6
        assert sum(c == "cudaMalloc" for c in calls) == 1
        assert_same(lat.download(), run_checker("port", case, 3), ctx=name)


@pytest.mark.parametrize("steps", [3, 4])
def test_given_back_after_any_number_of_steps(gpu_lib, steps):
    """T and U lie in the buffers after an odd number of steps."""
    from multiphaselb_b200 import Lattice
    case = channel(512, 384)
    got = []
    for limit in (False, True):
        with Lattice(case, path=abi.PATH_OPERATORS) as lat:
            lat.upload_case()
            lat.initialize()
            created = lat.info()["device_bytes"]
            lat.step(steps)
            lat.sync()
            held = lat.info()["device_bytes"]
            assert 0 <= held - created - 48 * case.n < 6 * 256
            if limit:
                with Nearly(170 * case.n):
                    lat.snapshot(pdfs=True)
                    lat.snapshot_wait()
                assert lat.info()["device_bytes"] == created + 192 * case.n
            lat.step(2)
            got.append(lat.download())
    for k in got[0]:
        assert np.array_equal(got[0][k], got[1][k]), k
