"""A batched cooperative PCG launch takes the kernel that carries the forms of its systems (the caller's CSR, packed
with 2- or 4-byte columns, streamed past the caches, any mixture): every solution and status is bit for bit that of
the solo solve."""
import ctypes as C
from functools import lru_cache

import pytest
import torch

from jspsr import _lib as L
from test_gpu_pcg_packed import batch_item, residual, system

pytestmark = pytest.mark.gpu
TOL = 1e-8


@lru_cache(maxsize=None)
def cached(n, per_row, seed):
    return system(n, per_row, seed)


# c: CSR, p: packed with 2-byte columns, w: with 4-byte ones, s: packed and larger than the streaming threshold
KINDS = {"c": (False, 0), "p": (True, 0), "w": (True, 1), "s": (True, 0)}


@pytest.mark.parametrize("kinds", ["p", "pp", "ww", "pw", "ps", "cc", "cp", "cpws", "ppppcc"])
@pytest.mark.parametrize("mode", [L.PCG_MIXED, L.PCG_FP64])
def test_batch_equals_solo(kinds, mode):
    jobs = []
    for k, kind in enumerate(kinds):
        packed, wide = KINDS[kind]
        m = cached(300001, 60, 1) if kind == "s" else cached(*((5003, 30), (20000, 61), (811, 4))[k % 3], 2 + k)
        blocks = 100 if kind == "s" else 3 + k                     # a block count: never a cluster
        jobs.append((m, wide, blocks, packed))
    items = [batch_item(m, mode, w, b, packed=p) for m, w, b, p in jobs]
    arr = (L.PcgBatchItem * len(items))(*[i[0] for i in items])
    L.call("ngs_pcg_solve_batch", arr, len(items), L.stream())
    for (m, w, b, p), (_, x, keep) in zip(jobs, items):
        assert int(keep[-1][1]) == 0 and residual(m, x) <= 1.01 * TOL
        solo, y, kept = batch_item(m, mode, w, b, packed=p)
        L.call("ngs_pcg_solve", C.byref(solo.sys), C.byref(solo.cfg), solo.ws, solo.ws_bytes, solo.info_dev,
               solo.resid_dev, L.stream())
        assert torch.equal(x, y) and torch.equal(keep[-1], kept[-1])
