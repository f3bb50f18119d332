"""Iterative refinement of the mixed mode on ill-conditioned systems whose values FP32 does not hold: scaled and shifted
Laplacians, where the recurrence's residual and the true one part during an inner solve.  Every solve reaches its
tolerance in the true FP64 residual, alone (a cluster or the grid), packed, and in a batch."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp
import torch

from jspsr import _lib as L
from test_gpu_pcg_packed import batch_item, residual

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


def laplacian(dims, shift, seed):
    """S (sum of the axes' second differences + shift) S with a random diagonal S, and a random right-hand side."""
    rng = np.random.default_rng(seed)
    n = int(np.prod(dims))
    a = shift * sp.identity(n)
    for d, m in enumerate(dims):
        e = np.ones(m - 1)
        t = sp.diags([np.concatenate([[0], e]) + np.concatenate([e, [0]]), -e, -e], [0, 1, -1])
        a = a + sp.kron(sp.kron(sp.identity(int(np.prod(dims[:d]))), t), sp.identity(int(np.prod(dims[d + 1:]))))
    s = sp.diags(1 + rng.uniform(-0.3, 0.3, n))
    a = (s @ a @ s).tocsr()
    a.sort_indices()
    rows = np.repeat(np.arange(n), np.diff(a.indptr))
    T = lambda v, t: torch.from_numpy(np.ascontiguousarray(v)).to(DEV, t)      # noqa: E731
    return dict(n=n, nnz=a.nnz, ptr=T(a.indptr, torch.int64), rows=T(rows, torch.int64), cols=T(a.indices, torch.int32),
                vals=T(a.data, torch.float64), diag=T(np.flatnonzero(rows == a.indices), torch.int64),
                b=T(rng.normal(size=n), torch.float64))


CASES = [((300,), 1e-6, 1e-10), ((60, 60), 1e-5, 1e-10), ((40, 40, 40), 1e-4, 1e-7), ((40, 40, 40), 1e-4, 1e-10),
         ((300, 300), 1e-6, 1e-7)]


@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("dims,shift,tol", CASES)
def test_true_residual_reaches_the_tolerance(dims, shift, tol, packed):
    m = laplacian(dims, shift, len(dims))
    for batch in (1, 2):
        items = [batch_item(m, L.PCG_MIXED, 0, 0, packed=packed) for _ in range(batch)]
        for item, _, _ in items:
            item.cfg.tol, item.cfg.max_iter, item.cfg.replace_every = tol, 19000, 0
        if batch == 1:
            item = items[0][0]
            L.call("ngs_pcg_solve", C.byref(item.sys), C.byref(item.cfg), item.ws, item.ws_bytes, item.info_dev,
                   item.resid_dev, L.stream())
        else:
            arr = (L.PcgBatchItem * 2)(*[i[0] for i in items])
            L.call("ngs_pcg_solve_batch", arr, 2, L.stream())
        for _, x, keep in items:
            assert int(keep[-1][1]) == 0, keep[-1].tolist()
            assert residual(m, x) <= 1.01 * tol
