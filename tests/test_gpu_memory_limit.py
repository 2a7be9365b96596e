"""Lattices on a nearly full device: what a failed call leaves behind."""
import gc

import pytest

from multiphaselb_b200 import abi, cases

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
