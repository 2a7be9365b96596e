"""Lattices on a nearly full device: what a failed call leaves behind."""
import gc

import numpy as np
import pytest

from multiphaselb_b200 import abi, cases, mesh
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


def channel(nx, ny):
    """A thermal channel around a disc: no box, so the operator path."""
    m = mesh.channel_with_cylinder(nx, ny, nx / 2 - 0.5, ny / 2.5, ny / 5.0)
    col = cases.column_case(nx, ny)
    keep = np.array([x + nx * y for x, y, _ in m.points.tolist()])
    tc = col.meta["Tc"]
    f = dict(col.f, bc_type=[abi.BC_BOUNCEBACK] * 3, bc_value=np.zeros((3, 3)))
    g = dict(col.g, bc_type=[abi.BC_FIXEDT] * 3, bc_value=np.array([[0.86 * tc, 0, 0], [0.84 * tc, 0, 0], [0.87 * tc, 0, 0]]))
    return mesh.mesh_case(m, "channel", col.eos, f, g, col.rho[keep], col.U[keep], col.T[keep],
                          meta=dict(Tc=tc, box=False))


def walls3d():
    c = cases.bubble_case(abi.D3Q15, 16, 4.0, 3.0, 0.75, dims=(193, 121, 167))
    c.nb, c.points, c.patches, c.patch_names = cases.box_mesh(abi.D3Q15, c.dims, (False, True, False))
    c.periodic = (False, True, False)
    c.f = dict(c.f, bc_type=[abi.BC_BOUNCEBACK] * len(c.patches), bc_value=np.zeros((len(c.patches), 3)))
    return cases.perturbed(c, du=1e-3)


# bytes a node left once the lattice has stepped: the snapshot of all fields needs
# 8 (6 + 2 Q), 192 and 288; the table kernels' buffers are 48 and 8
@pytest.mark.parametrize("make,kw,left", [(lambda: channel(1024, 768), dict(path=abi.PATH_OPERATORS), 170),
                                          (walls3d, dict(path=abi.PATH_FUSED, tile_config=6), 284)])
def test_table_buffers_go_before_a_call_fails(gpu_lib, make, kw, left):
    """A snapshot that fits only without the table kernels' buffers is taken, and
    the steps after it go on as if nothing had happened."""
    import torch
    from multiphaselb_b200 import Lattice
    case = make()

    def run(limit):
        with Lattice(case, **kw) as lat:
            lat.upload_case()
            lat.initialize()
            lat.step(3)
            lat.sync()
            held = lat.info()["device_bytes"]
            if limit:
                with Nearly(left * case.n):
                    lat.snapshot(pdfs=True)
                    snap = lat.snapshot_wait()
            else:
                lat.snapshot(pdfs=True)
                snap = lat.snapshot_wait()
            assert (lat.info()["device_bytes"] < held + 8 * case.n * (6 + 2 * case.Q)) == limit
            lat.step(3)
            torch.cuda.synchronize()
            return snap, lat.download()

    (want_snap, want), (snap, got) = run(False), run(True)
    for k in want_snap:
        assert np.array_equal(snap[k], want_snap[k]), k
    for k in want:
        assert np.array_equal(got[k], want[k]), k


def test_captured_table_steps_keep_their_scratch(gpu_lib):
    """A graph of the caller's that holds steps on the table candidate writes to its
    scratch at every replay: a call that lacks memory fails, the scratch stays."""
    import torch
    from multiphaselb_b200 import Lattice, MplbError
    case = walls3d()
    with Lattice(case, path=abi.PATH_FUSED, tile_config=6) as lat:
        lat.upload_case()
        lat.initialize()
        lat.step(6)
        want = lat.download()
    s = torch.cuda.Stream()
    with Lattice(case, path=abi.PATH_FUSED, tile_config=6, stream=s.cuda_stream) as lat:
        lat.upload_case()
        lat.initialize()
        lat.step(2)
        lat.sync()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            lat.step(2)
        held = lat.info()["device_bytes"]
        with Nearly(284 * case.n):
            with pytest.raises(MplbError) as e:
                lat.snapshot(pdfs=True)
            assert e.value.code == abi.E_CUDA
            assert lat.info()["device_bytes"] == held
            with torch.cuda.stream(s):
                graph.replay()
                graph.replay()
            torch.cuda.synchronize()
        got = lat.download()
        del graph
    for k in want:
        assert np.array_equal(got[k], want[k]), k


def test_tuner_needs_no_memory(gpu_lib):
    """The tuner times the table candidate on memory that the handle has; without
    the scratch that stepping on it takes, the lattice keeps its best tile."""
    from multiphaselb_b200 import Lattice
    case = walls3d()
    with Lattice(case, path=abi.PATH_FUSED) as lat:  # also loads every kernel that the second handle runs
        lat.upload_case()
        lat.initialize()
        lat.step(3)
        want = lat.download()
    with Lattice(case, path=abi.PATH_FUSED) as lat:
        lat.upload_case()
        lat.initialize()
        held = lat.info()["device_bytes"]
        with Nearly(4 * case.n):
            lat.step(3)
            info = lat.info()
            assert info["tile_ms"][5] > 0 and info["tile_config"] != 5
            assert info["device_bytes"] == held
        got = lat.download()
    for k in want:
        assert np.array_equal(got[k], want[k]), k
