"""Terms of an ``AdditiveBasis`` system in the kernels of ``csrc/learned.cu``: values at points, stiffness of voxel
pairs, divergence of voxel data and their derivatives, each one launch that reads the coefficients by voxel id and
adds into what the term belongs to.

They take the bases and tensors that ``AdditiveTerms.of`` accepts; everything else (other bases, components, types,
devices, overridden integrals, deterministic mode: the sums here go through atomics) keeps the torch form.
"""
from __future__ import annotations

import ctypes as C

import torch

from .. import _lib as L
from . import tables as TB
from .additive_components import Bezier, Power, SinPeaks, Sinusoid

MOST = 32            # components the kernels take
AXES_CHUNK = 1 << 20  # rows of coefficients gathered at once (ten components: 120 MB)


def component_table(components):
    """The components as ``ngs_basis_comps``, or None where one is not among the kernels'."""
    if not 0 < len(components) <= MOST:
        return None
    t = L.BasisComps()
    t.count = len(components)
    for k, c in enumerate(components):
        if type(c) is Power and type(c.power) is int and 0 <= c.power <= 64:
            t.kind[k], t.a[k] = L.COMP_POWER, c.power
        elif type(c) in (SinPeaks, Sinusoid) and all(type(v) in (int, float) for v in (c.beta, c.gamma)):
            t.kind[k], t.a[k], t.b[k] = L.COMP_SIN, c.beta, c.gamma
        elif type(c) is Bezier:
            t.kind[k] = L.COMP_BEZIER
        else:
            return None
    return t


def axes_table(components, xyz, coeffs, ids):
    """The components for ``ngs_basis_axes`` on these tensors, or None (the torch form)."""
    if not (xyz.is_cuda and coeffs.device == ids.device == xyz.device and xyz.dtype == coeffs.dtype == torch.float32 and
            xyz.dim() == 2 and xyz.shape[1] == 3 and coeffs.dim() == 2 and coeffs.shape[1] == 3 * len(components) and
            ids.dtype in (torch.int64, torch.int32) and ids.shape == xyz.shape[:1]):
        return None
    return component_table(components)


class AdditiveTerms:
    def __init__(self, basis, comps, dev):
        self.basis, self.comps, self.dev = basis, comps, dev

    @staticmethod
    def of(basis, shapes, feats_list, normals_list):
        """The terms for these shapes, or None where a tensor or the basis needs the torch form."""
        from .additive import AdditiveBasis
        from .hermite_ns import AdditiveHermite
        cls = type(basis)
        if not issubclass(cls, AdditiveBasis) or torch.are_deterministic_algorithms_enabled():
            return None
        if any(getattr(cls, m) is not getattr(AdditiveBasis, m) for m in
               ("evaluate", "integrate_deriv_deriv_product", "integrate_const_deriv_product", "_buf")):
            return None
        if cls.feature_to_coefficient not in (AdditiveBasis.feature_to_coefficient, AdditiveHermite.feature_to_coefficient):
            return None
        comps = component_table(basis.components)
        if comps is None:
            return None
        dev = shapes[0].levels[shapes[0].order[0]].level.device
        if dev.type != "cuda":
            return None

        def plain(t, shape):
            return t is not None and t.device == dev and t.dtype == torch.float32 and tuple(t.shape) == shape

        for shape, feats, normals in zip(shapes, feats_list, normals_list):
            order = shape.order
            if any(not plain(feats.get(d), (shape.levels[d].n, basis.get_feature_size())) for d in order):
                return None
            if any(dd not in shape.levels or not plain(normals.get(dd), (shape.levels[dd].n, 3))
                   for dd in shape.data_levels):
                return None
            if any(rel.dtype != torch.float32 for g in shape.levels.values()
                   for rel in [g.slot_rel] + [p[2] for p in g.cross.values()] + [p[2] for p in g.data.values()]):
                return None
            if max(order) - min(order) >= basis.n_multiples:
                return None
            for m in range(max(order) - min(order) + 1):
                ff = basis._buf(f"ff_{m}", dev)
                if ff.dtype != torch.float32 or not L.load().ngs_basis_pairs_fit(comps.count, ff.shape[-1]):
                    return None
        return AdditiveTerms(basis, comps, dev)

    def coefficients(self, feat):
        c = self.basis.feature_to_coefficient(feat)
        assert c.dtype == torch.float32 and c.shape == (feat.shape[0], 3 * self.comps.count)
        return c.contiguous()

    # ------------------------------------------------------------------ points
    def phi(self, geo, coef):
        n = geo.pt_rows.shape[0]
        out = torch.empty((n, 27), dtype=torch.float32, device=self.dev)
        L.call("ngs_basis_phi", C.byref(self.comps), L.ptr(coef), L.ptr(geo.pt_rows), L.ptr(geo.pt_local), n, L.ptr(out),
               L.stream())
        return out

    def phi_grad(self, geo, coef, lam, x, pa, pb, gcoef):
        L.call("ngs_basis_phi_grad", C.byref(self.comps), L.ptr(coef), L.ptr(geo.pt_rows), L.ptr(geo.pt_local),
               geo.pt_rows.shape[0], L.ptr(lam), L.ptr(x), L.ptr(pa), L.ptr(pb), L.ptr(gcoef), L.stream())

    def point_field(self, phi, geo, x):
        out = torch.empty(phi.shape[0], dtype=torch.float64, device=self.dev)
        L.call("ngs_point_sum64", L.ptr(phi), L.ptr(geo.pt_rows), phi.shape[0], L.ptr(x), L.ptr(out), L.stream())
        return out

    def point_spread(self, phi, geo, w, scale, out):
        L.call("ngs_point_spread64", L.ptr(phi), L.ptr(geo.pt_rows), phi.shape[0], L.ptr(w), float(scale), L.ptr(out),
               L.stream())

    # ------------------------------------------------------------------ pairs
    def _pairs(self, geo_s, geo_t, cs, ct):
        """The stiffness term of the pairs of a level (geo_s is geo_t) or towards a coarser one, and the tensors
        it reads."""
        M = geo_t.stride // geo_s.stride
        m = TB.ratio_log2(M)
        ff, dd = (self.basis._buf(f"{k}_{m}", self.dev).contiguous() for k in ("ff", "dfdf"))
        sid, tid, rel = (geo_s.slot_row, geo_s.cols, geo_s.slot_rel) if geo_s is geo_t else geo_s.cross[geo_t.depth]
        sid, tid, rel = sid.contiguous(), tid.contiguous(), rel.contiguous()
        t = L.BasisPairTerm()
        t.ff, t.dd, t.cs, t.ct = ff.data_ptr(), dd.data_ptr(), cs.data_ptr(), ct.data_ptr()
        t.sid, t.tid, t.rel, t.pairs = sid.data_ptr(), tid.data_ptr(), rel.data_ptr(), sid.shape[0]
        t.fscale, t.dscale, t.add = geo_s.stride, 1.0 / geo_s.stride, 1.5 * M + 0.5
        t.C, t.R, t.tid32 = self.comps.count, ff.shape[-1], int(tid.dtype == torch.int32)
        return t, (ff, dd, sid, tid, rel)

    def stiffness(self, geo, coef):
        """FP64 value of every CSR slot."""
        t, keep = self._pairs(geo, geo, coef, coef)
        out = torch.empty(geo.nnz, dtype=torch.float64, device=self.dev)
        t.out = out.data_ptr()
        L.call("ngs_basis_pairs", C.byref(t), 0, L.stream())
        return out

    def couple(self, geo_s, geo_t, cs, ct, x, y, transposed):
        """y[s] -= value x[t] of every pair (transposed: y[t] -= value x[s])."""
        t, keep = self._pairs(geo_s, geo_t, cs, ct)
        t.x, t.y, t.transposed = x.data_ptr(), y.data_ptr(), int(transposed)
        L.call("ngs_basis_pairs", C.byref(t), 0, L.stream())

    def pairs_grad(self, geo_s, geo_t, cs, ct, lam, x, gs, gt):
        t, keep = self._pairs(geo_s, geo_t, cs, ct)
        t.lam, t.xs = lam.data_ptr(), x.data_ptr()
        t.gs, t.gt = (g.data_ptr() if g is not None else None for g in (gs, gt))
        L.call("ngs_basis_pairs", C.byref(t), 1, L.stream())

    # ------------------------------------------------------------------ divergence
    def _divergence(self, geo, dd, coef, data):
        v, tid, rel = (a.contiguous() for a in geo.data[dd])
        ds, ts = 1 << dd, geo.stride
        t = L.BasisDivTerm()
        if ts >= ds:
            M = ts // ds
            fk, dk, t.scale, t.mul, t.add = "f", "df", ds, 1.0, (3 * M - 1) / 2.0
        else:
            M = ds // ts
            fk, dk, t.scale, t.mul, t.add = "finv", "dfinv", ts, M, M / 2 + 0.5
        m = TB.ratio_log2(M)
        tables = [[self.basis._buf(f"{k}_{i}_{m}", self.dev).contiguous() for i in range(self.comps.count)] for k in (fk, dk)]
        for i in range(self.comps.count):
            t.f[i], t.df[i] = tables[0][i].data_ptr(), tables[1][i].data_ptr()
        t.C, t.len = self.comps.count, tables[0][0].shape[0]
        t.coef, t.data, t.rel, t.vid, t.tid = coef.data_ptr(), data.data_ptr(), rel.data_ptr(), v.data_ptr(), tid.data_ptr()
        t.pairs = v.shape[0]
        return t, (v, tid, rel, tables)

    def divergence(self, geo, dd, coef, data, b):
        data = data.contiguous()
        t, keep = self._divergence(geo, dd, coef, data)
        t.b = b.data_ptr()
        L.call("ngs_basis_divergence", C.byref(t), 0, L.stream())

    def divergence_grad(self, geo, dd, coef, data, lam, gcoef, gdata):
        data = data.contiguous()
        t, keep = self._divergence(geo, dd, coef, data)
        t.lam = lam.data_ptr()
        t.gcoef, t.gdata = (g.data_ptr() if g is not None else None for g in (gcoef, gdata))
        L.call("ngs_basis_divergence", C.byref(t), 1, L.stream())
