"""The one-cluster FP64 CG of small CSR systems (fem_pcg) against scipy's
direct solve, at the sizes where its split can go wrong: fewer rows than CTAs,
the edges of a warp block and of each lanes-per-row range, the largest system
it takes and the first that is left to the grid-wide kernel, a row as long as
the system, and rows too many or too long for its shared memory (declined on
the device).

The matrices are symmetric with a diagonal of one plus the row's absolute sum, so
A >= I and the 2-norm error is at most ||r|| <= rtol ||b||; A <= 2 max(diag) I
gives ||b|| <= 2 max(diag) ||x||, hence a relative error of at most
2 max(diag) rtol, checked with a factor of 2 for the rounding of the recursive
residual.
"""

import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spl
import torch

from torchfem_gb300 import _lib

pytestmark = pytest.mark.gpu


def _system(n, kind):
    rng = np.random.default_rng(n)
    if kind == "dense":
        A = sp.csr_matrix(rng.uniform(-1, 1, (n, n)))
    else:
        offs = [k for k in ([1, 2, 3, 60, 61, 62] if kind == "stencil" else [1, 2, 7, 40]) if k < n]
        i = np.concatenate([np.arange(n - k) for k in offs] + [np.zeros(0, dtype=np.int64)])
        j = np.concatenate([np.arange(k, n) for k in offs] + [np.zeros(0, dtype=np.int64)])
        if kind == "arrow":  # one row and column hold every unknown
            i, j = np.concatenate([i, np.full(n, n // 2)]), np.concatenate([j, np.arange(n)])
        A = sp.coo_matrix((rng.uniform(-1, 1, len(i)), (i, j)), shape=(n, n)).tocsr()
    A = A + A.T
    A.setdiag(0.0)
    d = 1.0 + np.asarray(abs(A).sum(1)).ravel()
    A = (A + sp.diags(d)).tocsr()
    A.sort_indices()
    return A, d, rng.standard_normal(n)


@pytest.mark.parametrize("n,kind", [
    (1, "band"), (5, "band"), (31, "band"), (33, "arrow"), (129, "band"), (1600, "band"), (1601, "arrow"),
    (3201, "stencil"), (6401, "stencil"), (16000, "stencil"), (16384, "band"), (16385, "band"),
    (300, "dense"), (1500, "dense"), (9001, "arrow"),
])
def test_small_system_solution(cuda, n, kind):
    A, d, b = _system(n, kind)
    lib = _lib.load()
    t = lambda a, dt: torch.tensor(a, dtype=dt, device=cuda)  # noqa: E731
    row_ptr, col = t(A.indptr, torch.int64), t(A.indices, torch.int32)
    val, dinv, bt = t(A.data, torch.float64), t(1.0 / d, torch.float64), t(b, torch.float64)
    m = _lib.FemMatrix(_lib.FEM_FMT_CSR_F64, 1, n, n, row_ptr.data_ptr(), col.data_ptr(), val.data_ptr(),
                       dinv.data_ptr())
    ws = torch.empty(lib.fem_pcg_workspace_bytes(C.byref(m)), dtype=torch.uint8, device=cuda)
    x = torch.full((n,), float("nan"), dtype=torch.float64, device=cuda)
    info = _lib.FemSolveInfo()
    rtol = 1e-12
    args = (ws.data_ptr(), ws.numel(), C.byref(info), _lib.stream_handle(cuda))
    assert lib.fem_pcg(C.byref(m), bt.data_ptr(), x.data_ptr(), rtol, 10 * n, *args) == _lib.FEM_OK
    assert info.rel_residual <= rtol
    ref = np.asarray(spl.spsolve(A.tocsc(), b)).ravel()
    err = np.linalg.norm(x.cpu().numpy() - ref) / np.linalg.norm(ref)
    assert err <= 2 * 2 * d.max() * rtol, err
    # the iteration limit and a zero right-hand side
    if n > 100:
        assert lib.fem_pcg(C.byref(m), bt.data_ptr(), x.data_ptr(), rtol, 1, *args) == _lib.FEM_NOT_CONVERGED
        assert info.iterations == 1 and torch.isfinite(x).all()
    bt.zero_()
    assert lib.fem_pcg(C.byref(m), bt.data_ptr(), x.data_ptr(), rtol, 10 * n, *args) == _lib.FEM_OK
    assert info.iterations == 0 and not x.any()
    bt[n // 2] = float("nan")
    assert lib.fem_pcg(C.byref(m), bt.data_ptr(), x.data_ptr(), rtol, 10 * n, *args) == _lib.FEM_NONFINITE
