"""The screening Gram and right-hand sides over points grouped by cell, with shares long enough for every loop of a
warp's walk: several steps of 32 positions, runs carried over from step to step and cut at a share's end, points
without a voxel at a share's beginning, a count that no share divides, weights and a field.

Against one FP64 atomic per point: all terms are positive, so two orders of summing a row's m of them differ by less
than 2 m 2^-53 of the sum (Higham, first order); a dropped or doubled point shows as some 1 / m.
"""
import pytest
import torch

from jspsr import _lib as L

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


# shares of 43 and 29 positions, and their caps of 128 and 256
@pytest.mark.parametrize("n", [200_003, 2_000_003])
def test_grouped_equals_per_point(n):
    from jspsr import synthetic
    from jspsr.core.pipeline import Reconstruction
    xyz, nrm = (torch.from_numpy(a).to(DEV) for a in synthetic.torus(n=n))
    rec = Reconstruction(xyz, nrm, 1 / 64, 5, None).build_tree().assemble()
    g = torch.Generator(device=DEV).manual_seed(n)
    without = torch.rand(n, generator=g, device=DEV) < 0.01
    w = torch.rand(n, generator=g, device=DEV) + 0.5
    field = torch.rand(n, generator=g, device=DEV) + 0.5
    longest, st = 0, L.stream()
    for lv in rec.levels:
        rows = torch.where(without[:, None], -1, lv.rows).contiguous()
        phi = torch.where(without[:, None], 0.0, lv.phi).contiguous()
        keys = torch.empty(n, dtype=torch.int64, device=DEV)
        L.call("ngs_point_cell_keys", L.ptr(rows), n, L.ptr(keys), st)
        keys, order = torch.sort(keys)
        assert int(keys[0]) == -1
        longest = max(longest, int(torch.unique_consecutive(keys, return_counts=True)[1][1:].max()))
        flat = rows.reshape(-1)
        m = torch.bincount(flat[flat >= 0].long(), minlength=lv.n).double()
        for weights in (None, w):
            a, b = torch.zeros(2, lv.nnz, dtype=torch.float64, device=DEV)
            L.call("ngs_screen_gram", L.ptr(rows), L.ptr(phi), n, L.ptr(weights), L.ptr(lv.masks), L.ptr(lv.rowptr), 0.75,
                   L.ptr(a), st)
            L.call("ngs_screen_gram_grouped", L.ptr(rows), L.ptr(phi), n, L.ptr(weights), L.ptr(order), L.ptr(keys),
                   L.ptr(lv.masks), L.ptr(lv.rowptr), 0.75, L.ptr(b), st)
            row = torch.repeat_interleave(torch.arange(lv.n, device=DEV), lv.rowptr[1:] - lv.rowptr[:-1])
            # the products of a term differ by a few roundings besides
            assert ((a - b).abs() <= (2 * m[row] + 8) * 2.0 ** -53 * a).all()
        for weights, f in ((None, None), (w, None), (None, field), (w, field)):
            a, b = torch.zeros(2, lv.n, dtype=torch.float64, device=DEV)
            if f is None:
                L.call("ngs_screen_rhs", L.ptr(rows), L.ptr(phi), n, L.ptr(weights), 0.75, L.ptr(a), st)
            else:
                L.call("ngs_correction_screen", L.ptr(rows), L.ptr(phi), n, L.ptr(weights), L.ptr(f), -0.75, L.ptr(a), st)
            L.call("ngs_screen_rhs_grouped", L.ptr(rows), L.ptr(phi), n, L.ptr(weights), L.ptr(f), L.ptr(order),
                   L.ptr(keys), 0.75, L.ptr(b), st)
            assert ((a - b).abs() <= (2 * m + 8) * 2.0 ** -53 * a.abs()).all()
    assert longest > 4 * 256                                   # runs longer than any share
