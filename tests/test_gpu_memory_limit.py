"""Lattices on a nearly full device: what a failed call leaves behind."""
import gc

import pytest

from multiphaselb_b200 import abi, cases
from tests.helpers import mymrt

pytestmark = pytest.mark.gpu


class Nearly:
    """Holds device memory so that about `free` bytes are left to others."""

    def __init__(self, free):
        import torch
        self.torch = torch
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        have = torch.cuda.mem_get_info()[0]
        assert have > free
        self.block = torch.empty(have - free, dtype=torch.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *a):
        del self.block
        gc.collect()
        self.torch.cuda.empty_cache()


def test_call_after_a_failed_create(gpu_lib):
    """The allocation that failed is reported by its own call only."""
    from multiphaselb_b200 import Lattice, MplbError
    big, small = cases.column_case(1024, 2048), cases.column_case(32, 64)
    with Lattice(small) as lat, Nearly(400 * big.n):
        with pytest.raises(MplbError) as e:
            Lattice(big)
        assert e.value.code == abi.E_CUDA
        lat.upload_case()
        lat.initialize()
        lat.step(2)
        lat.download()


def test_failed_create_gives_everything_back(gpu_lib):
    """A myMRT column of 2 Mi nodes needs 478 bytes a node.  With less, its create
    fails at one allocation or another, and leaves the device as it was."""
    import torch
    from multiphaselb_b200 import Lattice, MplbError
    c = cases.column_case(1024, 2048)
    c.g = mymrt(abi.D2Q9, [abi.BC_FIXEDT] * 2, c.g["bc_value"])
    with Lattice(c, path=abi.PATH_FUSED):  # what a create loads is on the device from here on
        pass
    failed = 0
    for per_node in range(400, 500, 8):
        with Nearly(per_node * c.n):
            left = []
            for _ in range(3):
                try:
                    Lattice(c, path=abi.PATH_FUSED).close()
                except MplbError as e:
                    assert e.code == abi.E_CUDA
                    failed += 1
                left.append(torch.cuda.mem_get_info()[0])
            assert left[0] == left[1] == left[2], (per_node, left)
    assert 3 <= failed < 39 and failed % 3 == 0, failed
