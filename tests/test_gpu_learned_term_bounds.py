"""Every kernel of the learned basis' terms by itself against the same sum in 64 bits, to its own rounding.

u = 2^-24.  First-order bounds (Higham) in units of the sum of the terms' magnitudes, which the same formula gives on
the absolute values of its factors: an axis' p or q of a pair is a sum of C sums of C products (2 C + 3 roundings), its
value a sum of three products of three of them (6 C + 16); a gradient holds two axes, the tables' C products and its
g (6 C + 20), and an FP32 sum of m of them m more.  A divergence's p or q is a sum of C products (C + 3).  Component
values are within eight roundings.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)
U = 2.0 ** -24
MOST = 30_000                        # pairs of a gradient


@pytest.fixture(scope="module", params=[1, 8, 10])
def problem(request):
    from jspsr import synthetic
    from jspsr.bases.additive import AdditiveBasis
    from jspsr.bases.additive_components import Bezier, Power, SinPeaks
    from jspsr.bases.additive_terms import AdditiveTerms
    from jspsr.core import galerkin as G
    from jspsr.core.hashtree import HashTree
    from jspsr.core.learned import LearnedStep
    C = request.param
    comps = [Bezier()] + [SinPeaks(k + 1) for k in range(2)] + [Power(p) for p in range(7)]
    basis = AdditiveBasis(comps[:C], [1.0] + [0.0] * (C - 1)).to(DEV)
    xyz, nrm, q, tgt = [torch.from_numpy(a).to(DEV) for a in synthetic.learned_problem(500, 10, seed=5)[:4]]
    st = LearnedStep(xyz, nrm, q, tgt, voxel_size=1 / 32, min_density=None, basis=basis).build()
    shape = G.ShapeGeometry.build(st.tree, HashTree.DECODER, st.depth - 1, 0, list(range(st.depth)), xyz, 4.0, 0.1, 3)
    g = torch.Generator(device=DEV).manual_seed(C)

    def rand(*s, dtype=torch.float32):
        return torch.randn(*s, generator=g, device=DEV, dtype=torch.float64).to(dtype)
    coef = {d: rand(shape.levels[d].n, 3 * C) for d in shape.order}
    vec = {d: (rand(shape.levels[d].n, dtype=torch.float64), rand(shape.levels[d].n, dtype=torch.float64)) for d in shape.order}
    data = {d: rand(shape.levels[d].n, 3) for d in shape.order}
    feats = {d: torch.zeros(shape.levels[d].n, basis.get_feature_size(), device=DEV) for d in shape.order}
    terms = AdditiveTerms.of(basis, [shape], [feats], [data])
    assert terms is not None and len(shape.order) > 1
    return basis, C, shape, terms, coef, vec, data


def close(got, ref, mag, bound):
    assert got.shape == ref.shape and bool(((got.double() - ref).abs() <= bound * mag + 1e-36).all())


def count(ids, n):
    return torch.bincount(ids.long(), minlength=n).double()


def pair_sum(term, ff, dd, cs, ct, mag):
    """64-bit value of every pair of an `ngs_basis_pair_term`'s numbers (magnitudes of its terms)."""
    sid, tid, rel, fscale, dscale, add = term
    a = torch.abs if mag else (lambda v: v)
    at = torch.round(rel + add).long()
    ok = (at >= 0) & (at < ff.shape[-1])
    at = at.clamp(0, ff.shape[-1] - 1)
    C = ff.shape[0]
    s, t = a(cs.double())[sid].view(-1, C, 3), a(ct.double())[tid].view(-1, C, 3)
    p, q = (torch.where(ok, torch.einsum("stpa,psa,pta->pa", a(tab.double())[:, :, at] * scale, s, t), 0.0)
            for tab, scale in ((ff, fscale), (dd, dscale)))
    return q[:, 0] * p[:, 1] * p[:, 2] + p[:, 0] * q[:, 1] * p[:, 2] + p[:, 0] * p[:, 1] * q[:, 2]


def pair_terms(problem):
    basis, C, shape, terms, coef, vec, data = problem
    for d in shape.order:
        for e in [d] + sorted(shape.levels[d].cross):
            geo, ge = shape.levels[d], shape.levels[e]
            t, (ff, dd, sid, tid, rel) = terms._pairs(geo, ge, coef[d], coef[e])
            yield d, e, ff, dd, (sid, tid.long(), rel, t.fscale, t.dscale, t.add)


def test_pair_values(problem):
    basis, C, shape, terms, coef, vec, data = problem
    seen = 0
    for d, e, ff, dd, term in pair_terms(problem):
        def values(mag):
            return torch.cat([pair_sum(tuple(v[k:k + MOST] for v in term[:3]) + term[3:], ff, dd, coef[d], coef[e], mag)
                              for k in range(0, len(term[0]), MOST)])
        if not len(term[0]):
            continue
        seen += 1
        ref, mag = values(False), values(True)
        geo, ge, bound = shape.levels[d], shape.levels[e], (6 * C + 16) * U
        if d == e:
            close(terms.stiffness(geo, coef[d]), ref, mag, bound)
            continue
        s, t = term[:2]
        for transposed, x, out, n in ((False, vec[e][0][t], s, geo.n), (True, vec[d][0][s], t, ge.n)):
            y = torch.zeros(n, dtype=torch.float64, device=DEV)
            terms.couple(geo, ge, coef[d], coef[e], vec[d][0] if transposed else vec[e][0], y, transposed)
            close(y, y.new_zeros(n).index_add_(0, out, -ref * x), y.new_zeros(n).index_add_(0, out, mag * x.abs()), bound)
    assert seen > 2


def test_pair_gradients(problem):
    basis, C, shape, terms, coef, vec, data = problem
    for d, e, ff, dd, term in pair_terms(problem):
        if d == e or not len(term[0]):
            continue                                          # same level: the same kernel, into one array
        geo, ge = shape.levels[d], shape.levels[e]
        whole = geo.cross[e]
        geo.cross[e] = tuple(v[:MOST] for v in whole[:3])
        s, t, rel = term[0][:MOST], term[1][:MOST], term[2][:MOST]
        gs, gt = torch.zeros_like(coef[d]), torch.zeros_like(coef[e])
        terms.pairs_grad(geo, ge, coef[d], coef[e], vec[d][0], vec[e][1], gs, gt)
        geo.cross[e] = whole
        got = {}
        for mag in (False, True):
            cs, ct = (c.double().abs().requires_grad_(True) if mag else c.double().requires_grad_(True) for c in (coef[d], coef[e]))
            w = -(vec[d][0][s] * vec[e][1][t])
            v = pair_sum((s, t, rel) + term[3:], ff, dd, cs, ct, mag)
            got[mag] = torch.autograd.grad((v * (w.abs() if mag else w)).sum(), (cs, ct))
        for k, (g, ids) in enumerate(((gs, s), (gt, t))):
            close(g, got[False][k], got[True][k], (6 * C + 20 + count(ids, g.shape[0]))[:, None] * U)


def divergence_sum(tables, term, coef, data, mag):
    """64-bit value of every pair (data voxel, target) (magnitudes of its terms)."""
    v, t, rel, mul, add, scale = term
    a = torch.abs if mag else (lambda x: x)
    at = torch.round(rel * mul + add).long()
    c, n = a(coef).double()[t].view(len(t), -1, 3), a(-data).double()[v]
    p = sum(c[:, k] * (a(tables[0][k].double())[at] * scale) for k in range(len(tables[0])))
    q = sum(c[:, k] * a(tables[1][k].double())[at] for k in range(len(tables[1])))
    return n[:, 0] * q[:, 0] * p[:, 1] * p[:, 2] + n[:, 1] * p[:, 0] * q[:, 1] * p[:, 2] + n[:, 2] * p[:, 0] * p[:, 1] * q[:, 2]


def test_divergence_and_gradients(problem):
    basis, C, shape, terms, coef, vec, data = problem
    for d in shape.order:
        geo = shape.levels[d]
        for dd in shape.data_levels:
            t, (v, tid, rel, tables) = terms._divergence(geo, dd, coef[d], data[dd])
            term = (v, tid, rel, t.mul, t.add, t.scale)
            if not len(v):
                continue
            b = torch.zeros(geo.n, dtype=torch.float64, device=DEV)
            terms.divergence(geo, dd, coef[d], data[dd], b)
            lam = vec[d][0]
            ref, mag = (divergence_sum(tables, term, coef[d], data[dd], m) for m in (False, True))
            z = torch.zeros(geo.n, dtype=torch.float64, device=DEV)
            close(b, z.index_add(0, tid, ref), z.index_add(0, tid, mag), (3 * (C + 3) + 5) * U)
            gcoef, gdata = torch.zeros_like(coef[d]), torch.zeros_like(data[dd])
            terms.divergence_grad(geo, dd, coef[d], data[dd], lam, gcoef, gdata)
            got = {}
            for m in (False, True):
                ins = [(x.double().abs() if m else x.double()).requires_grad_(True) for x in (coef[d], data[dd])]
                s = divergence_sum(tables, term, *ins, m) * (lam.abs() if m else lam)[tid]
                got[m] = [g.abs() if m else g for g in torch.autograd.grad(s.sum(), ins)]
            close(gcoef, got[False][0], got[True][0], (2 * (C + 3) + 16 + count(tid, geo.n))[:, None] * U)
            close(gdata, got[False][1], got[True][1], (3 * (C + 3) + 8 + count(v, len(data[dd])))[:, None] * U)


def test_points(problem):
    basis, C, shape, terms, coef, vec, data = problem
    for d in shape.order:
        geo, (lam, x) = shape.levels[d], vec[d]
        n = geo.pt_rows.shape[0]
        rows, there = geo.pt_rows.clamp(min=0).long(), geo.pt_rows >= 0
        q = torch.stack([torch.sin((c.beta * geo.pt_local + c.gamma).double()) if hasattr(c, "beta")
                         else c.evaluate(geo.pt_local.double()) for c in basis.components], 2)         # [n, 27, C, 3]
        # a component's own rounding is relative to its largest value on the support
        size = q.abs().clamp(min=1)

        def value(c, comps):
            return torch.where(there, (c[rows].view(n, 27, C, 3) * comps).sum(2).prod(2), 0.0)
        c64 = coef[d].double()
        phi = terms.phi(geo, coef[d])
        close(phi, value(c64, q), value(c64.abs(), size), 3 * (C + 9) * U)
        # sums over the slots, and back, of the kernel's own values: 64 bits
        term = torch.where(there, phi.double() * x[rows], 0.0)
        close(terms.point_field(phi, geo, x), term.sum(1), term.abs().sum(1), 64 * 2.0 ** -53)
        w, out = torch.randn(n, dtype=torch.float64, device=DEV), torch.zeros_like(x)
        terms.point_spread(phi, geo, w, 0.3, out)
        term = torch.where(there, 0.3 * phi.double() * w[:, None], 0.0).reshape(-1)
        ids = rows.reshape(-1)
        m = count(ids[there.reshape(-1)], geo.n)
        close(out, torch.zeros_like(x).index_add(0, ids, term), torch.zeros_like(x).index_add(0, ids, term.abs()),
              (2 * m + 4) * 2.0 ** -53)
        pa, pb = torch.randn(2, n, dtype=torch.float64, device=DEV)
        got = torch.zeros_like(coef[d])
        terms.phi_grad(geo, coef[d], lam, x, pa, pb, got)
        up = lam[rows] * pa[:, None] + x[rows] * pb[:, None]
        grads = []
        for c, comps, u in ((c64, q, up), (c64.abs(), size, up.abs())):
            c = c.clone().requires_grad_(True)
            grads.append(torch.autograd.grad((value(c, comps) * u).sum(), c)[0])
        close(got, grads[0], grads[1], (2 * (C + 9) + 16 + m)[:, None] * U)
