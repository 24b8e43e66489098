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
