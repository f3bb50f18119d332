"""The box tree of ``jspsr.sdfgen`` at the sizes where its levels fill up (32 points to a leaf, 32
children to a node), with ties, repeated points, fewer points than neighbours, and queries far off.

Points and queries lie on an integer lattice of extent 512, so that every squared distance is an exact
FP32 number: distances and indices (nearest first, ties to the smaller index) must equal a brute force.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


def brute(q, xyz, k):
    d2 = ((q[:, None, :] - xyz[None, :, :]) ** 2).sum(-1)
    idx = np.argsort(d2, axis=1, kind="stable")[:, :k]               # stable: ties to the smaller index
    return idx, np.take_along_axis(d2, idx, 1)


@pytest.mark.parametrize("n", [1, 5, 31, 32, 33, 1023, 1024, 1025, 32768, 32769])
@pytest.mark.parametrize("k", [1, 8, 32])
def test_tree_equals_brute_force(n, k):
    from jspsr import sdfgen
    rng = np.random.default_rng(n * 37 + k)
    xyz = rng.integers(0, 512, (n, 3))
    if n > 4:
        xyz[n // 2:n // 2 + n // 4] = xyz[:n // 4]                   # repeated points
        xyz[:, 2] = np.where(rng.random(n) < 0.5, 7, xyz[:, 2])      # half of them in one plane
    q = np.concatenate([rng.integers(0, 512, (61, 3)), xyz[rng.integers(0, n, 30)], rng.integers(-700, 1200, (30, 3))])
    idx, d2 = sdfgen.knn(torch.from_numpy(q).float().to(DEV), torch.from_numpy(xyz).float().to(DEV), k)
    m = min(n, k)
    want_idx, want_d2 = brute(q, xyz, m)
    np.testing.assert_array_equal(idx.cpu().numpy()[:, :m], want_idx)
    np.testing.assert_array_equal(d2.cpu().numpy()[:, :m], want_d2.astype(np.float32))
    assert (idx[:, m:] == -1).all() and torch.isinf(d2[:, m:]).all()


def test_one_place_and_infinite_queries():
    """All points in one place (a bounding box of no extent), and queries at infinity: every distance ties,
    and the smallest indices win."""
    from jspsr import sdfgen
    xyz = torch.full((100, 3), 0.25, device=DEV)
    q = torch.tensor([[0.25, 0.25, 0.25], [1.0, 0.25, 0.25], [float("inf"), 0.0, 0.0]], device=DEV)
    idx, d2 = sdfgen.knn(q, xyz, 8)
    assert torch.equal(idx, torch.arange(8, dtype=torch.int32, device=DEV).expand(3, 8))
    assert torch.equal(d2[:, 0], torch.tensor([0.0, 0.5625, float("inf")], device=DEV))


def test_tree_equals_grid_walk():
    """The grid walk of the C ABI (ngs_knn_*) and the tree give the same neighbours and distances."""
    from jspsr import _lib as L, sdfgen, synthetic
    xyz, nrm, _ = synthetic.superquadrics(7001, k=2, seed=3)
    rng = np.random.default_rng(3)
    q = (xyz[rng.integers(0, len(xyz), 5000)] + rng.normal(0, 0.02, (5000, 3))).astype(np.float32)
    X, N, Q = (torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).to(DEV) for a in (xyz, nrm, q))
    h = 0.05
    inv = np.float32(1 / h)
    lo = np.floor(xyz.min(0) * inv).astype(np.int64)
    hi = np.floor(xyz.max(0) * inv).astype(np.int64)
    g, words = L.make_grid(lo, hi - lo + 1, 1, DEV)
    n, st = len(xyz), L.stream()
    L.call("ngs_knn_mark_cells", g, L.ptr(X), n, inv, st)
    cnt = torch.empty(1, dtype=torch.int64, device=DEV)
    ws = L.grid_finalize(g, words, cnt)
    nc = int(cnt.item())
    cell, count = torch.empty(n, dtype=torch.int32, device=DEV), torch.zeros(nc, dtype=torch.int32, device=DEV)
    L.call("ngs_knn_bucket", g, L.ptr(X), n, inv, L.ptr(cell), L.ptr(count), st)
    start = torch.empty(nc + 1, dtype=torch.int64, device=DEV)
    L.scan(count, out=start[:nc], total=start[nc:])
    cursor, order = torch.zeros(nc, dtype=torch.int32, device=DEV), torch.empty(n, dtype=torch.int32, device=DEV)
    L.call("ngs_knn_scatter", L.ptr(cell), n, L.ptr(start), L.ptr(cursor), L.ptr(order), st)
    idx, d2 = torch.empty((5000, 8), dtype=torch.int32, device=DEV), torch.empty((5000, 8), device=DEV)
    sdf = torch.empty(5000, device=DEV)
    L.call("ngs_knn_sdf", g, L.ptr(start), L.ptr(order), L.ptr(X), L.ptr(N), L.ptr(Q), 5000, inv, h, 8, 0.02, L.ptr(idx),
           L.ptr(d2), L.ptr(sdf), st)
    ti, td, ts = sdfgen.PointIndex(X, N).query(Q, 8, stdv=0.02)
    assert torch.equal(ti, idx) and torch.equal(td, d2) and torch.equal(ts, sdf)
    del ws
