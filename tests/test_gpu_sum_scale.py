"""The grid-wide sums of the persistent CG where a quantity falls far in one
iteration: their fixed point's scale comes from the last sum of the same quantity.

The matrix is diagonal with entries 1 and 1 + 2^-47 in turn, no preconditioner, b = 1.
First iteration: p.q = n (1 + 2^-48), alpha = 1 - 2^-48 up to rounding, r = -+2^-48, and
r.r falls by 2^-96; then p.q by as much, of which a CTA has less than a hundredth.
The second step solves the system, its residual below 2^-48 * 2^-47 |b|.  So with rtol
= 1e-15 (2^-49.8) CG takes exactly two iterations, and x_i d_i - 1 is the rounding of
two additions and two products of numbers near one: at most 2^-50.
"""

import ctypes as C

import pytest
import torch

from torchfem_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block", [0, 1, 2, 3])
@pytest.mark.parametrize("rows", [16416, 32768, 131072])
def test_falling_sums(cuda, block, rows):
    lib = _lib.load()
    n = rows * max(block, 1)
    d = torch.ones(n, dtype=torch.float64, device=cuda)
    d[1::2] += 2.0**-47
    one = torch.ones(n, dtype=torch.float64, device=cuda)
    col = torch.arange(rows, dtype=torch.int32, device=cuda)
    if block == 0:  # scalar CSR, more rows than the one-cluster kernel takes
        ptr, val = torch.arange(n + 1, dtype=torch.int64, device=cuda), d
    else:  # sliced blocks, one slot-row a slice: [component][row]
        ptr = torch.arange(0, rows + 1, 32, dtype=torch.int64, device=cuda)
        val = torch.zeros(rows // 32, block, block, 32, dtype=torch.float64, device=cuda)
        for i in range(block):
            val[:, i, i] = d.reshape(-1, 32, block)[:, :, i]
    m = _lib.FemMatrix(_lib.FEM_FMT_SELL_F64 if block else _lib.FEM_FMT_CSR_F64, max(block, 1), n, rows,
                       ptr.data_ptr(), col.data_ptr(), val.data_ptr(), one.data_ptr())
    ws = torch.empty(lib.fem_pcg_workspace_bytes(C.byref(m)), dtype=torch.uint8, device=cuda)
    x = torch.full((n,), float("nan"), dtype=torch.float64, device=cuda)
    info = _lib.FemSolveInfo()
    before = lib.fem_get_cg_path()
    lib.fem_set_cg_path(1)
    try:
        rc = lib.fem_pcg(C.byref(m), one.data_ptr(), x.data_ptr(), 1e-15, 50, ws.data_ptr(), ws.numel(),
                         C.byref(info), _lib.stream_handle(cuda))
    finally:
        lib.fem_set_cg_path(before)
    assert rc == _lib.FEM_OK and info.iterations == 2
    assert float((x * d - 1.0).abs().max()) <= 2.0**-50
