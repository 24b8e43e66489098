"""Host logic of DeviceMesh around the sliced layout, with a stand-in for the
library (no GPU)."""

import pytest
import torch

from torchfem_gb300 import _device, _lib


class FakeLib:
    """Records the calls it gets; every call succeeds."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def call(*args):
            self.calls.append(name)
            if name == "fem_sell_layout":
                args[2]._obj.value = 64  # n_slots
            return 0

        return call


@pytest.fixture
def dm(monkeypatch):
    dm = object.__new__(_device.DeviceMesh)
    dm.lib, dm.device, dm.blocks = FakeLib(), torch.device("cpu"), _lib.FemBlocks()
    dm.n_nod, dm.d, dm.n_dofs, dm.nnz = 40, 1, 40, 100
    dm.row_ptr = torch.zeros(41, dtype=torch.int64)
    dm._sell = None

    class Stream:
        def synchronize(self):
            dm.lib.calls.append(("sync", dm._sell))

    monkeypatch.setattr(_lib, "stream_handle", lambda device: 0)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: Stream())
    return dm


def test_layout_is_complete_before_it_is_shown(dm):
    layout = dm.sell()
    columns = dm.lib.calls.index("fem_sell_columns")
    assert dm.lib.calls[columns + 1:] == [("sync", None)]
    assert dm.sell() is layout and len(dm.lib.calls) == columns + 2


@pytest.mark.parametrize("allocations", [0, 1, 2, 3, None])
def test_without_memory_for_the_sliced_copy_cg_keeps_csr(dm, monkeypatch, allocations):
    monkeypatch.setattr(dm, "CG_CLUSTER_NNZ", {1: 0}, raising=False)
    monkeypatch.setattr(dm, "_ws", lambda n: torch.zeros(1, dtype=torch.uint8), raising=False)
    sysm = _device.LinearSystem(dm, "fp64")
    sysm.val, sysm.precond = torch.zeros(100, dtype=torch.float64), torch.ones(40, dtype=torch.float64)
    sysm.matrix = _lib.FemMatrix(_lib.FEM_FMT_CSR_F64, 1, 40, 40, None, None, None, None)
    given = []

    def empty(n, dtype):
        if allocations is not None and len(given) >= allocations:
            raise torch.OutOfMemoryError("no memory left")
        given.append(torch.zeros(int(n), dtype=dtype))
        return given[-1]

    monkeypatch.setattr(dm, "_empty", empty, raising=False)
    # the layout's bases and columns, then the values
    fits = allocations is None or allocations >= 3
    for _ in range(2):
        m = dm.cg_matrix(sysm)
        assert m.format == (_lib.FEM_FMT_SELL_F64 if fits else _lib.FEM_FMT_CSR_F64)
    assert fits or m is sysm.matrix
