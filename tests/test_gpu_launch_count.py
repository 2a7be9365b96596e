"""mplb_info.kernel_launches counts the kernels that a step launches."""
import pytest

from multiphaselb_b200 import abi
from tests.captured import captured_kernels
from tests.helpers import small_cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,tile,per_step", [("walls_d3q15", 6, 2), ("walls_d3q15", 3, 1), ("my_column_d2q9", 1, 2),
                                                ("my_column_d2q9", 11, 1), ("column_d2q9", 1, 1)])
def test_launches_of_a_step(gpu_lib, name, tile, per_step):
    """The table candidate launches two a step, a myMRT tile its pre-pass and the
    step, the march and the other tiles one."""
    import torch
    from multiphaselb_b200 import Lattice
    stream = torch.cuda.Stream()
    with Lattice(small_cases()[name], path=abi.PATH_FUSED, tile_config=tile, stream=stream.cuda_stream) as lat:
        lat.upload_case()
        lat.initialize()
        lat.step(1)
        lat.sync()
        before = lat.info()["kernel_launches"]
        kernels = captured_kernels(stream, lambda: lat.step(4))
        assert lat.info()["kernel_launches"] - before == len(kernels) == 4 * per_step, kernels
