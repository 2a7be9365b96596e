"""Batch and Lattice handles are destroyed in the library's order, the batch
before its lattices, whatever order Python drops the objects in (garbage
collection finalises a cycle's objects in no useful order; a batch destroyed
after its lattices would use a stream that no longer exists).  A stand-in for
the library records the calls; no GPU needed."""
import gc

import pytest

import multiphaselb_b200 as mp
from multiphaselb_b200 import abi, cases


class FakeLibrary:
    def __init__(self):
        self.calls = []
        self.handles = 0

    def _new(self, out):
        self.handles += 1
        out._obj.value = self.handles
        return 0

    def mplb_gpu_create(self, mesh, eos, f, g, opts, out):
        return self._new(out)

    def mplb_batch_create(self, arr, n, opts, out):
        return self._new(out)

    def mplb_gpu_destroy(self, h):
        self.calls.append("lattice")
        return 0

    def mplb_batch_destroy(self, h):
        self.calls.append("batch")
        return 0

    def mplb_batch_step(self, h, n):
        return 0 if h and h.value else -1

    def mplb_gpu_last_error(self):
        return b"NULL batch"


@pytest.fixture
def fake(monkeypatch):
    lib = FakeLibrary()
    monkeypatch.setattr(mp, "load_library", lambda *a: lib)
    return lib


def make(n=3):
    case = cases.bubble_case(abi.D2Q9, 8, 2.0, 2.0, 0.8)
    lats = [mp.Lattice(case) for _ in range(n)]
    return lats, mp.Batch(lats)


def test_cycle_of_lattices_and_batch(fake):
    lats, batch = make()
    cycle = dict(lats=lats, batch=batch)  # as a script's globals
    cycle["self"] = cycle
    del lats, batch, cycle
    gc.collect()
    assert fake.calls == ["batch"] + ["lattice"] * 3


def test_lattice_closed_first(fake):
    lats, batch = make()
    lats[1].close()
    assert fake.calls == ["batch", "lattice"]
    with pytest.raises(mp.MplbError):
        batch.step(1)
    batch.close()
    for lat in lats:
        lat.close()
    assert fake.calls == ["batch"] + ["lattice"] * 3


def test_batch_closed_first_and_dropped(fake):
    lats, batch = make()
    batch.close()
    assert fake.calls == ["batch"]
    second = mp.Batch(lats)
    del batch, second  # no reference of a lattice keeps a batch alive
    assert fake.calls == ["batch", "batch"]
    del lats
    gc.collect()
    assert fake.calls == ["batch", "batch"] + ["lattice"] * 3
