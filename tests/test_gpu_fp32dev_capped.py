"""The register-capped FP32 2D kernel with inner tiles (16 x 8 tiles, eight blocks
per SM), which lattices of more than 1036 tiles of 32 x 8 step on: every field
against FP64 within the bounds of the other FP32 kernels."""
import pytest

from multiphaselb_b200 import abi, cases
from tests.captured import captured_kernels
from tests.helpers import run_gpu
from tests.test_gpu_fp32dev import BIG, SMALL, TOL_BIG, TOL_SMALL, rel_err, run32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", ["column", "bubble"])
def test_capped_kernel_close_to_fp64(gpu_lib, shape):
    """256 x 1100 (1104 tiles, the last row of them partial) and 549 x 541 (1224,
    partial on both axes)."""
    import torch
    from multiphaselb_b200 import Lattice
    case = (cases.column_case(256, 1100, amp=1e-3) if shape == "column"
            else cases.perturbed(cases.bubble_case(abi.D2Q9, 512, 80.0, 5.0, 0.8, dims=(549, 541)), du=1e-3))
    assert ((case.dims[0] + 31) // 32) * ((case.dims[1] + 7) // 8) > 1036
    want, _ = run_gpu(case, 10, path=abi.PATH_FUSED)
    got = run32(case, 10)[-1]
    stream = torch.cuda.Stream()
    with Lattice(case, precision=abi.FP32_DEV, stream=stream.cuda_stream) as lat:
        lat.upload_case()
        lat.initialize()
        lat.step(2)
        lat.sync()
        kernels = captured_kernels(stream, lambda: lat.step(2))
    # tile, flow, heat, programs, EMIT, blocks per SM
    assert len(kernels) == 2 and all(k == "k_fused32_d2q9" and a[:2] == (16, 8) and a[6] == 8 for k, a in kernels), kernels
    errs = {k: rel_err(got[k], want[k]) for k in BIG + SMALL if not (k == "g" and case.g is None)
            and not (k in ("S", "T") and case.g is None)}
    print(shape, errs)
    for k, e in errs.items():
        assert e <= (TOL_BIG if k in BIG else TOL_SMALL), (shape, k, e)
