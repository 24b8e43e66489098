"""Which FP64 CSR systems the one-cluster CG takes, by the launches of a solve: one
kernel there, a start and at least one more on the grid-wide path.  Edges: the
rows of a cluster, the shared memory, and the longest row (160 entries to a lane, one
lane per row from 257 rows a CTA on, at most eight below).  Both sides solve: the
matrices are A = diag(1 + row sums) + symmetric entries in [-1, 1], A >= I, so that
||b - A x|| <= rtol ||b|| up to the rounding of A x, below 2^-53 ||A||_1 ||x|| times
the entries of a row, and ||A||_1 ||x|| <= 2 max(diag) ||b||.
"""

import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp
import torch

from torchfem_gb300 import _lib

pytestmark = pytest.mark.gpu


def _matrix(n, offsets, longest=0):
    """Entries on the given side diagonals, and one last row of `longest` entries."""
    rng = np.random.default_rng(n + longest)
    i = np.concatenate([np.arange(n - k) for k in offsets])
    j = np.concatenate([np.arange(k, n) for k in offsets])
    if longest:
        keep = j != n - 1
        c = rng.choice(n - 1, longest - 1, replace=False)
        i, j = np.concatenate([i[keep], c]), np.concatenate([j[keep], np.full(longest - 1, n - 1)])
    A = sp.coo_matrix((rng.uniform(-1, 1, len(i)), (i, j)), shape=(n, n)).tocsr()
    A = A + A.T
    d = 1.0 + np.asarray(abs(A).sum(1)).ravel()
    A = (A + sp.diags(d)).tocsr()
    A.sort_indices()
    if longest:
        assert A.indptr[-1] - A.indptr[-2] == longest
    return A, d


WIDE = [1, 2, 3, 60, 61, 62, 120, 121]
CASES = {
    # name: (rows, side diagonals, entries of the last row, taken by the cluster)
    "one row": (1, [], 0, True),
    "most rows": (16384, [], 0, True),
    "a row too many": (16385, [], 0, False),
    "a CTA with too many rows": (16380, [16000], 0, False),
    "most entries": (3900, list(range(1, 39)), 0, True),
    "too many entries": (4000, list(range(1, 50)), 0, False),
    "too wide a window": (16000, [1, 2, 3, 4, 8000, 15000], 0, False),
    "single lanes, longest": (6000, WIDE, 160, True),
    "single lanes, too long": (6000, WIDE, 161, False),
    "eight lanes, longest": (1500, WIDE, 1280, True),
    "eight lanes, too long": (1500, WIDE, 1281, False),
}


@pytest.mark.parametrize("name", CASES)
def test_path(cuda, name):
    n, offsets, longest, taken = CASES[name]
    A, d = _matrix(n, offsets, longest) if offsets else (sp.diags(np.linspace(1.0, 2.0, n)).tocsr(),
                                                         np.linspace(1.0, 2.0, n))
    lib = _lib.load()
    t = lambda a, dt: torch.tensor(a, dtype=dt, device=cuda)  # noqa: E731
    row_ptr, col = t(A.indptr, torch.int64), t(A.indices, torch.int32)
    val, dinv = t(A.data, torch.float64), t(1.0 / d, torch.float64)
    b = np.random.default_rng(0).standard_normal(n)
    bt = t(b, torch.float64)
    m = _lib.FemMatrix(_lib.FEM_FMT_CSR_F64, 1, n, n, row_ptr.data_ptr(), col.data_ptr(), val.data_ptr(),
                       dinv.data_ptr())
    ws = torch.empty(lib.fem_pcg_workspace_bytes(C.byref(m)), dtype=torch.uint8, device=cuda)
    x = torch.full((n,), float("nan"), dtype=torch.float64, device=cuda)
    info = _lib.FemSolveInfo()
    before = lib.fem_launch_count()
    rtol = 1e-10
    assert lib.fem_pcg(C.byref(m), bt.data_ptr(), x.data_ptr(), rtol, 10 * n, ws.data_ptr(), ws.numel(),
                       C.byref(info), _lib.stream_handle(cuda)) == _lib.FEM_OK
    assert (lib.fem_launch_count() - before <= 2) == taken
    row = int(np.diff(A.indptr).max())
    bound = (rtol + 2.0**-53 * row * 2 * d.max()) * np.linalg.norm(b)
    assert np.linalg.norm(b - A @ x.cpu().numpy()) <= bound
