"""Diagonals of any CSR for the direct-solve replacement: rows shorter and longer than eight entries, unsorted and
repeated entries (summed in 64 bits: three values, order-independent to 2 ulp), rows without a diagonal (1 / 0), and
the calls that are refused."""
import numpy as np
import pytest
import torch

from jspsr import _lib as L
from jspsr import ext

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("n", [1, 31, 33, 4097])
def test_inverse_diagonal(n):
    rng = np.random.default_rng(n)
    counts = rng.integers(0, 40, n)
    rows = np.repeat(np.arange(n), counts)
    cols = np.where(rng.random(len(rows)) < 0.1, rows, rng.integers(0, n, len(rows)))
    vals = rng.uniform(0.5, 2, len(rows))
    ptr = torch.from_numpy(np.concatenate([[0], np.cumsum(counts)])).to(DEV)
    inv = torch.empty(n, device=DEV)
    c, v = torch.from_numpy(cols.astype(np.int32)).to(DEV), torch.from_numpy(vals).to(DEV)
    L.call("ngs_csr_diag_inv", L.ptr(ptr), L.ptr(c), L.ptr(v), n, L.ptr(inv), L.stream())
    d = np.zeros(n)
    np.add.at(d, rows[cols == rows], vals[cols == rows])
    with np.errstate(divide="ignore"):
        ref = (1 / d).astype(np.float32)
    assert np.array_equal(np.isinf(ref), np.isinf(inv.cpu().numpy()))
    np.testing.assert_allclose(inv.cpu().numpy(), ref, rtol=2.0 ** -22)


def test_refused_calls():
    ptr, cols = torch.tensor([0, 1, 2], device=DEV), torch.tensor([0, 1], device=DEV)
    vals, b = torch.ones(2, device=DEV), torch.ones(2, device=DEV)
    assert torch.allclose(ext.solve_cusparse(ptr, cols, vals, b, 1e-12), b)
    for bad in ((ptr[:2], cols, vals, b), (ptr, cols[:1], vals[:1], b), (torch.tensor([0, 3, 2], device=DEV), cols, vals, b),
                (ptr, cols, vals[:1], b)):
        with pytest.raises(Exception):
            ext.solve_cusparse(*bad, 1e-12)
