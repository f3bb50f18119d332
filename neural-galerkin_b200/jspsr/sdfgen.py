"""Signed distance from oriented points and exact k-nearest neighbours on the GPU.

Drop-in for the reference's ``ext.sdf_from_points(queries, ref_xyz, ref_normal, nb_points, stdv)``
(``ext/__init__.py:11-16``, ``ext/sdfgen/sdf_from_points.cu:70-116``), the ground truth of the
training loop (``models/full_net.py:135-142``).  The reference builds a CUDA k-d tree per call; here
the reference points are ordered along a Morton curve by a counting sort and boxed 32 to a leaf in a
32-ary tree, and one warp per query visits the boxes nearest first until no other can hold one of its
k nearest points, then votes the sign (``csrc/knn.cu``).
"""
from __future__ import annotations

import torch

from . import _lib as L


class PointIndex:
    """Reference points in a box tree for repeated nearest-neighbour queries.  ``cell``, the cell size of
    a grid index, has no effect: the tree sizes itself."""

    def __init__(self, ref_xyz: torch.Tensor, ref_normal: torch.Tensor = None, cell: float = None):
        L.require_cuda(ref_xyz, "ref_xyz")
        self.xyz = ref_xyz.detach().float().contiguous()
        self.normal = None if ref_normal is None else ref_normal.detach().float().contiguous()
        n = self.xyz.shape[0]
        if n == 0:
            raise ValueError("no reference points")
        lib, dev = L.load(), self.xyz.device
        self.tree = torch.empty(lib.ngs_knn_tree_bytes(n), dtype=torch.uint8, device=dev)
        scratch = torch.empty(lib.ngs_knn_tree_scratch_bytes(n), dtype=torch.uint8, device=dev)
        L.call("ngs_knn_tree_build", L.ptr(self.xyz), n, L.ptr(self.tree), self.tree.numel(), L.ptr(scratch),
               scratch.numel(), L.stream())

    def query(self, queries: torch.Tensor, k: int, stdv: float = None, want_knn: bool = True):
        """(indices int32 [Q, k], squared distances [Q, k], signed distance [Q] or None)."""
        L.require_cuda(queries, "queries")
        q = queries.detach().float().contiguous()
        nq, dev = q.shape[0], q.device
        idx = torch.empty((nq, k), dtype=torch.int32, device=dev) if want_knn else None
        d2 = torch.empty((nq, k), dtype=torch.float32, device=dev) if want_knn else None
        sdf = None
        if stdv is not None:
            if self.normal is None:
                raise ValueError("signed distances need the reference normals")
            sdf = torch.empty(nq, dtype=torch.float32, device=dev)
        L.call("ngs_knn_tree_query", L.ptr(self.tree), self.tree.numel(), L.ptr(self.xyz), self.xyz.shape[0],
               L.ptr(self.normal), L.ptr(q), nq, int(k), float(stdv if stdv is not None else 0.0), L.ptr(idx),
               L.ptr(d2), L.ptr(sdf), L.stream())
        return idx, d2, sdf


def knn(queries: torch.Tensor, ref_xyz: torch.Tensor, k: int):
    """Exact k nearest reference points of every query: (indices [Q, k], squared distances [Q, k]),
    nearest first, ties broken by the smaller index."""
    idx, d2, _ = PointIndex(ref_xyz).query(queries, k)
    return idx, d2


def sdf_from_points(queries: torch.Tensor, ref_xyz: torch.Tensor, ref_normal: torch.Tensor, nb_points: int,
                    stdv: float) -> torch.Tensor:
    """Signed distance of every query from the oriented reference points: magnitude from the nearest
    point (distance to its tangent plane within ``stdv``, Euclidean beyond), sign by the majority of
    the ``nb_points`` nearest normals (``ext/sdfgen/sdf_from_points.cu:31-68``)."""
    _, _, sdf = PointIndex(ref_xyz, ref_normal).query(queries, nb_points, stdv=stdv, want_knn=False)
    return sdf
