"""A snapshot's work on the device up to its copy, the rebuild of the reference
state included, does not wait for the previous snapshot's transfer."""
import time

import pytest

from multiphaselb_b200 import abi, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("path", [abi.PATH_OPERATORS, abi.PATH_FUSED])
def test_rebuild_overlaps_the_transfer(gpu_lib, path):
    """1024 x 2048: a transfer of 100 MB takes 2 ms or more, a step and its
    rebuild 0.4 ms."""
    import torch
    from multiphaselb_b200 import Lattice
    case = cases.bubble_case(abi.D2Q9, 1024, 200.0, 5.0, 0.8, dims=(1024, 2048))
    with Lattice(case, path=path) as lat:
        lat.upload_case()
        lat.initialize()
        for _ in range(2):
            lat.step(1)
            lat.snapshot()
        lat.snapshot_wait()
        lat.sync()
        def run():
            for _ in range(3):
                lat.step(1)
                lat.snapshot()
            lat.snapshot_wait()

        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            time.sleep(0.05)
            run()
            torch.cuda.synchronize()
            time.sleep(0.05)
        events = sorted(prof.events(), key=lambda e: e.time_range.start)
        transfers = [e for e in events if "DtoH" in e.name and e.time_range.elapsed_us() > 500]
        # the rebuild: the last kernel of the handle before each snapshot's transposition
        kernels = [e for e in events if "k_" in e.name]
        rebuilds = [kernels[i - 1] for i, e in enumerate(kernels) if "k_soa_to_aos" in e.name]
        if len(transfers) != 3 or len(rebuilds) != 3:
            pytest.skip("the profiler's clock put events outside the profile, which drops them")
        for before, rebuild in zip(transfers[:2], rebuilds[1:]):
            assert rebuild.time_range.end < before.time_range.end, (before, rebuild)
