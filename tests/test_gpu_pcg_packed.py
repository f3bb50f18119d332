"""The PCG's packed matrix at the edges of its groups (four rows), units (eight entries a row) and batches
(8, 12 or 16 units), with rows of very different lengths in one group.

Every solve must reach its tolerance in the true FP64 residual (the mixed mode checks it; the FP64 mode stops
on the recurrence's, which drifts from the true one by rounding), the packed form must hold the CSR's entries
exactly, and the column width changes no bit of the solution.
"""
import ctypes as C

import numpy as np
import pytest
import torch

from jspsr import _lib as L

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)
TOL = 1e-8


def system(n, per_row, seed, reach=30000, dense_row=False):
    """Symmetric, strictly diagonally dominant, |column - row| <= reach; sorted columns."""
    rng = np.random.default_rng(seed)
    m = n * per_row // 2
    r = rng.integers(0, n, m)
    c = np.clip(r + rng.integers(1, min(n, reach) + 1, m), 0, n - 1)
    if dense_row:
        k = min(n, reach + 1)
        c, r = np.concatenate([c, np.arange(1, k)]), np.concatenate([r, np.zeros(k - 1, np.int64)])
    keep = r != c
    key = np.unique(r[keep].astype(np.int64) * n + c[keep])
    r, c = key // n, key % n
    v = rng.uniform(-1, 1, len(r))
    off = np.zeros(n)
    np.add.at(off, r, np.abs(v))
    np.add.at(off, c, np.abs(v))
    rows = np.concatenate([r, c, np.arange(n)])
    cols = np.concatenate([c, r, np.arange(n)])
    vals = np.concatenate([v, v, 1.05 * off + 0.1])
    o = np.lexsort((cols, rows))
    rows, cols, vals = rows[o], cols[o], vals[o].astype(np.float32).astype(np.float64) * (1 + 1e-9)
    ptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    T = lambda a, t: torch.from_numpy(np.ascontiguousarray(a)).to(DEV, t)      # noqa: E731
    return dict(n=n, nnz=len(vals), ptr=T(ptr, torch.int64), rows=T(rows, torch.int64), cols=T(cols, torch.int32),
                vals=T(vals, torch.float64), diag=T(np.flatnonzero(rows == cols), torch.int64),
                b=T(rng.normal(size=n), torch.float64))


def pack(m, mode, wide):
    """Start of every group's units, values and column words."""
    groups = L.load().ngs_pcg_pack_groups(m["n"])
    units = torch.empty(groups, dtype=torch.int32, device=DEV)
    L.call("ngs_pcg_pack_count", L.ptr(m["ptr"]), m["n"], L.ptr(units), L.stream())
    start = torch.cat([torch.zeros(1, dtype=torch.int64, device=DEV), units.long().cumsum(0)])
    total = int(start[-1])
    vals = torch.empty(total * 32, dtype=torch.float64 if mode == L.PCG_FP64 else torch.float32, device=DEV)
    cols = torch.zeros(L.load().ngs_pcg_pack_col_words(m["n"], total, wide), dtype=torch.int32, device=DEV)
    L.call("ngs_pcg_pack_fill", L.ptr(m["ptr"]), L.ptr(m["cols"]), L.ptr(m["vals"]), m["n"], L.ptr(start), wide, mode,
           L.ptr(vals), L.ptr(cols), L.stream())
    return start, vals, cols


def solve(m, mode, wide, blocks=0):
    item, x64, keep = batch_item(m, mode, wide, blocks)
    L.call("ngs_pcg_solve", C.byref(item.sys), C.byref(item.cfg), item.ws, item.ws_bytes, item.info_dev, item.resid_dev,
           L.stream())
    info = keep[-1]
    assert int(info[1]) == 0, int(info[1])
    return x64


def batch_item(m, mode, wide, blocks=0, packed=True):
    start, vals, cols = pack(m, mode, wide)
    dinv = torch.empty(m["n"], device=DEV)
    L.call("ngs_csr_inv_diag", L.ptr(m["vals"]), L.ptr(m["diag"]), m["n"], L.ptr(dinv), L.stream())
    x32, x64 = torch.empty(m["n"], device=DEV), torch.zeros(m["n"], dtype=torch.float64, device=DEV)
    info = torch.zeros(4, dtype=torch.int64, device=DEV)
    resid = torch.zeros(2, dtype=torch.float64, device=DEV)
    item = L.PcgBatchItem()
    s, cfg = item.sys, item.cfg
    s.n, s.nnz, s.rowptr, s.cols, s.vals64 = m["n"], m["nnz"], m["ptr"].data_ptr(), m["cols"].data_ptr(), m["vals"].data_ptr()
    s.inv_diag, s.b64, s.x32, s.x64 = dinv.data_ptr(), m["b"].data_ptr(), x32.data_ptr(), x64.data_ptr()
    v32 = m["vals"].float()
    if packed:
        s.pk_start, s.pk_vals, s.pk_cols = start.data_ptr(), vals.data_ptr(), cols.data_ptr()
        s.pk_units, s.pk_wide = int(start[-1]), wide
    else:
        s.vals32 = v32.data_ptr()
    cfg.mode, cfg.max_iter, cfg.tol, cfg.res_fix = mode, 5000, TOL, 0
    cfg.replace_every, cfg.blocks, cfg.timeout_s = 50, blocks, 10.0
    nb = L.load().ngs_pcg_workspace_bytes(m["n"], mode)
    ws = torch.empty(nb, dtype=torch.uint8, device=DEV)
    item.ws, item.ws_bytes, item.info_dev, item.resid_dev = ws.data_ptr(), nb, info.data_ptr(), resid.data_ptr()
    return item, x64, (m, start, vals, cols, dinv, x32, v32, resid, ws, info)


def residual(m, x):
    y = torch.zeros_like(m["b"]).index_add_(0, m["rows"], m["vals"] * x[m["cols"].long()])
    return float(torch.linalg.norm(m["b"] - y) / torch.linalg.norm(m["b"]))


# group remainders, rows within one batch and over several (12, 16 units = 96, 128 entries), one block to many
SIZES = [(1, 0), (3, 2), (4, 2), (5, 4), (33, 8), (1001, 3), (4097, 90), (4098, 130), (40003, 30), (300001, 60)]


@pytest.mark.parametrize("n,per_row", SIZES)
@pytest.mark.parametrize("mode", [L.PCG_MIXED, L.PCG_FP64])
def test_solutions_and_column_widths(n, per_row, mode):
    m = system(n, per_row, n + mode)
    x = solve(m, mode, 0)
    assert residual(m, x) <= (TOL if mode == L.PCG_MIXED else 1.01 * TOL)
    assert torch.equal(x, solve(m, mode, 1))


@pytest.mark.parametrize("mode", [L.PCG_MIXED, L.PCG_FP64])
def test_one_long_row_and_few_blocks(mode):
    """A row of 20,000 entries beside rows of six; one block and three take all rows."""
    m = system(30000, 6, 3, reach=20000, dense_row=True)
    for wide, blocks in ((0, 0), (1, 0), (0, 1), (1, 3)):
        assert residual(m, solve(m, mode, wide, blocks)) <= 1.01 * TOL


@pytest.mark.parametrize("n,per_row", [(1, 0), (5, 4), (1003, 70)])
@pytest.mark.parametrize("wide", [0, 1])
def test_packed_entries(n, per_row, wide):
    m = system(n, per_row, 11)
    start, vals, cols = (t.cpu().numpy() for t in pack(m, L.PCG_FP64, wide))
    ptr, c, v = (m[k].cpu().numpy() for k in ("ptr", "cols", "vals"))
    for row in range(n):
        g, q = divmod(row, 4)
        units = int(start[g + 1] - start[g])
        u, lane = np.divmod(np.arange(units * 8), 8)
        lane = lane + 8 * q
        got_v = vals[(start[g] + u) * 32 + lane]
        if wide:
            got_c = cols[(start[g] + u) * 32 + lane]
        else:
            words = cols[((start[g] + g + 1) // 2 + u // 2) * 32 + lane]
            got_c = row + np.where(u % 2, words >> 16, (words << 16) >> 16)
        k = ptr[row + 1] - ptr[row]
        assert np.array_equal(got_v[:k], v[ptr[row]:ptr[row + 1]]) and np.array_equal(got_c[:k], c[ptr[row]:ptr[row + 1]])
        assert not got_v[k:].any() and (got_c[k:] == row).all()


@pytest.mark.parametrize("mode", [L.PCG_MIXED, L.PCG_FP64])
def test_clusters_of_a_batch_equal_solo_solves(mode):
    """Small systems of one batch share launches by cluster size and form (at most 16 a launch): every solution is
    bit for bit that of its solo solve, with forms and sizes mixed and a system without a batch partner."""
    lib = L.load()
    shapes = [(2000, 20)] * 18 + [(1, 0), (300, 5), (9001, 40), (9002, 40), (0, 0), (4000, 60)]
    systems = [system(n, per, 7 + k) for k, (n, per) in enumerate(shapes) if n]
    kinds = [(k % 5 == 4, k % 3 != 1) for k in range(len(systems))]                  # 4-byte columns, packed
    assert len({lib.ngs_pcg_cluster_size(m["n"], m["nnz"], mode) for m in systems}) > 2
    assert all(lib.ngs_pcg_cluster_size(m["n"], m["nnz"], mode) > 0 for m in systems)
    items = [batch_item(m, mode, int(w), packed=p) for m, (w, p) in zip(systems, kinds)]
    arr = (L.PcgBatchItem * len(items))(*[i[0] for i in items])
    L.call("ngs_pcg_solve_batch", arr, len(items), L.stream())
    for m, (w, p), (_, x, keep) in zip(systems, kinds, items):
        assert int(keep[-1][1]) == 0 and residual(m, x) <= 1.01 * TOL
        solo, y, kept = batch_item(m, mode, int(w), packed=p)
        L.call("ngs_pcg_solve", C.byref(solo.sys), C.byref(solo.cfg), solo.ws, solo.ws_bytes, solo.info_dev,
               solo.resid_dev, L.stream())
        assert torch.equal(x, y) and torch.equal(keep[-1], kept[-1])
