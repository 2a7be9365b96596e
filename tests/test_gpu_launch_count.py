"""mplb_info.kernel_launches counts the kernels that a step launches."""
import pytest

from multiphaselb_b200 import abi
from tests.helpers import small_cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,tile", [("walls_d3q15", 6), ("walls_d3q15", 3), ("my_column_d2q9", 1),
                                       ("my_column_d2q9", 11), ("column_d2q9", 1)])
def test_launches_are_the_profilers(gpu_lib, name, tile):
    """The table candidate launches two a step, a myMRT tile its pre-pass and the
    step, the march and the other tiles one."""
    import torch
    from multiphaselb_b200 import Lattice
    with Lattice(small_cases()[name], path=abi.PATH_FUSED, tile_config=tile) as lat:
        lat.upload_case()
        lat.initialize()
        lat.step(1)
        lat.sync()
        before = lat.info()["kernel_launches"]
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            lat.step(5)
            lat.sync()
            torch.cuda.synchronize()
        seen = [e for e in prof.events() if "k_" in e.name]
        assert lat.info()["kernel_launches"] - before == len(seen) > 0
