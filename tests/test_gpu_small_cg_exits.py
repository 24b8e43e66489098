"""Exits of the one-cluster FP64 CG at its first and at its later decisions, in
systems with so few rows that most warps of a CTA have none: those warps send no
share of a sum and have to leave the loop with the others all the same.

The matrices are diagonal with entries 1 and a in turn, no preconditioner and b =
s everywhere, n a power of two, so that the scalars are known.  First iteration:
p.q = s^2 n (1 + a) / 2, alpha = 2 / (1 + a), r = s (1 - alpha, 1 - a alpha).

a = -1: p.q = 0 at once.
a = 0: alpha = 2, r = s (-1, 1), beta = 1, p = s (0, 2), q = 0: p.q = 0 in the second
  iteration, with x = 2 s.
a = -1 + 2^-52, s = 2^460: alpha = 2^53, r of size 2^513: r.r overflows.
a = -1 + 2^-40, s = 2^450: r of size 2^491, r.r = n 2^982 is finite, p = beta p of
  size 2^532: p.q overflows in the second iteration.

Every product and sum above is exact or out of range, so the codes and counts hold
whatever the order of the sums.
"""

import ctypes as C

import pytest
import torch

from torchfem_gb300 import _lib

pytestmark = pytest.mark.gpu

EXITS = {
    "p.q zero": (-1.0, 1.0, _lib.FEM_BREAKDOWN, 0),
    "p.q zero later": (0.0, 1.0, _lib.FEM_BREAKDOWN, 1),
    "r.r overflows": (-1.0 + 2.0**-52, 2.0**460, _lib.FEM_NONFINITE, 1),
    "p.q overflows later": (-1.0 + 2.0**-40, 2.0**450, _lib.FEM_NONFINITE, 1),
}


@pytest.mark.parametrize("n", [2, 16, 64, 512, 2048, 4096])
@pytest.mark.parametrize("case", EXITS)
def test_exit(cuda, case, n):
    a, s, code, iterations = EXITS[case]
    lib = _lib.load()
    row_ptr = torch.arange(n + 1, dtype=torch.int64, device=cuda)
    col = torch.arange(n, dtype=torch.int32, device=cuda)
    val = torch.ones(n, dtype=torch.float64, device=cuda)
    val[1::2] = a
    one = torch.ones(n, dtype=torch.float64, device=cuda)
    m = _lib.FemMatrix(_lib.FEM_FMT_CSR_F64, 1, n, n, row_ptr.data_ptr(), col.data_ptr(), val.data_ptr(),
                       one.data_ptr())
    ws = torch.empty(lib.fem_pcg_workspace_bytes(C.byref(m)), dtype=torch.uint8, device=cuda)
    x = torch.full((n,), float("nan"), dtype=torch.float64, device=cuda)
    info = _lib.FemSolveInfo()
    args = (x.data_ptr(), 1e-12, 100, ws.data_ptr(), ws.numel(), C.byref(info), _lib.stream_handle(cuda))
    b = torch.full((n,), s, dtype=torch.float64, device=cuda)
    for _ in range(20):
        before = lib.fem_launch_count()
        assert lib.fem_pcg(C.byref(m), b.data_ptr(), *args) == code
        assert lib.fem_launch_count() - before <= 2  # the one-cluster kernel, nothing behind it
        assert info.iterations == iterations
    if case == "p.q zero later":
        assert torch.equal(x, 2.0 * b)
    val.fill_(4.0)
    assert lib.fem_pcg(C.byref(m), one.data_ptr(), *args) == _lib.FEM_OK
    assert info.iterations == 1 and torch.equal(x, 0.25 * one)
