"""The learned basis' terms in kernels against their torch form: one to twelve components (thirteen keep the torch
form), levels that carry normal data or not, with and without screening, gradients of features, of normals or both.

Solutions and gradients are compared norm-wise at 2e-3: both forms round FP32 pair values at about 1e-5 of a system
whose condition (Jacobi-scaled, screened) is of the order of 1e2; a missing or wrongly signed term is of order one.
Values per axis are compared with 64 bits at (C + 8) 2^-22 of the sum of the terms' magnitudes; a sine's argument
beta x + gamma is the FP32 one in both, as in the components' torch form (near a zero of the sine its rounding alone
exceeds any bound relative to the value).
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


def basis_of(name):
    from jspsr.bases.additive import AdditiveBasis
    from jspsr.bases.additive_components import Bezier, Power, SinPeaks
    from jspsr.bases.hermite_ns import AdditiveHermite
    if name == "bezier":
        return AdditiveBasis([Bezier()], [1.0])
    if name == "two":
        return AdditiveBasis([Bezier(), SinPeaks(1)], [1.0, 0.0])
    return AdditiveHermite(6, [SinPeaks(k + 1) for k in range(name - 7)], [0.0] * (name - 7))


@pytest.mark.parametrize("name", ["bezier", "two", 8, 10, 13])
@pytest.mark.parametrize("m", [0, 1, 85, (1 << 20) + 3])
def test_values_per_axis(name, m):
    from jspsr.bases.additive import EvalFunc
    b = basis_of(name)
    C = len(b.components)
    g = torch.Generator().manual_seed(m + C)
    n = 50
    x = (torch.rand((m, 3), generator=g) * 3 - 1.5).to(DEV)
    coef = torch.randn((n, 3 * C), generator=g).to(DEV).requires_grad_(True)
    ids = torch.randint(0, n, (m,), generator=g).to(DEV)
    r = torch.randn((m, 3), generator=g).to(DEV)
    f = EvalFunc.apply(x, coef, ids, b.components)
    got, = torch.autograd.grad((f * r).sum(), coef)
    q = torch.stack([torch.sin((c.beta * x + c.gamma).double()) if hasattr(c, "beta") else c.evaluate(x.double())
                     for c in b.components], 1)                                              # [m, C, 3]
    terms = q * coef.detach().double()[ids].view(m, C, 3)
    assert ((f - terms.sum(1)).abs() <= (C + 8) * 2.0 ** -22 * terms.abs().sum(1) + 1e-30).all()
    gr = (q * r.double()[:, None]).reshape(m, 3 * C)
    ref, mag = (torch.zeros((n, 3 * C), dtype=torch.float64, device=DEV).index_add_(0, ids, t) for t in (gr, gr.abs()))
    # sums of m / n terms in FP32: their rounding grows at most with the count
    assert ((got - ref).abs() <= (8 + m / n) * 2.0 ** -22 * mag + 1e-30).all()


@pytest.mark.parametrize("name,alpha,grads", [("bezier", 4.0, "both"), ("two", 0.0, "both"), (8, 4.0, "normals"),
                                              (10, 4.0, "both"), (10, 4.0, "features"), (10, 0.0, "normals"),
                                              (12, 4.0, "both"), (13, 4.0, "both")])
def test_solutions_and_gradients(name, alpha, grads, monkeypatch):
    from jspsr.bases.additive_terms import AdditiveTerms
    from jspsr.core import galerkin as G
    from jspsr.core.learned import LearnedStep
    from jspsr import synthetic
    from jspsr.core.hashtree import HashTree
    xyz, nrm, q, tgt = [torch.from_numpy(a).to(DEV) for a in synthetic.learned_problem(700, 10, seed=5)[:4]]
    basis = basis_of(name).to(DEV)
    st = LearnedStep(xyz, nrm, q, tgt, voxel_size=1 / 32, min_density=None, basis=basis).build()
    data_levels = [d for d in range(st.depth) if bool((st.tree.xyz_depth == d).any())]
    shape = G.ShapeGeometry.build(st.tree, HashTree.DECODER, st.depth - 1, 0, data_levels, xyz, alpha, 0.1, 3)
    feats0 = st.init_features(sigma=0.05)
    rng = torch.Generator().manual_seed(1)
    weights = {d: torch.randn(shape.levels[d].n, generator=rng).to(DEV) for d in shape.order}

    def run():
        n = nrm.clone().requires_grad_(grads != "features")
        f = {d: v.clone().requires_grad_(grads != "normals") for d, v in feats0.items()}
        x = G.galerkin_solve(basis, [shape], [f], [st.normal_data(n)])[0]
        inputs = ([n] if n.requires_grad else []) + [v for v in f.values() if v.requires_grad]
        return [x[d].detach() for d in shape.order] + list(
            torch.autograd.grad(sum((x[d] * weights[d]).sum() for d in x), inputs))

    used = []
    of = AdditiveTerms.of
    monkeypatch.setattr(AdditiveTerms, "of", staticmethod(lambda *a: used.append(of(*a)) or used[-1]))
    got = run()
    assert (used[0] is None) == (name == 13)
    monkeypatch.setattr(AdditiveTerms, "of", staticmethod(lambda *a: None))
    for a, b in zip(got, run()):
        assert torch.isfinite(a).all()
        assert float((a - b).norm()) <= 2e-3 * float(b.norm())


def test_deterministic_mode_keeps_the_torch_form():
    from jspsr.bases.additive_terms import AdditiveTerms
    torch.use_deterministic_algorithms(True)
    try:
        assert AdditiveTerms.of(basis_of(10), [], [], []) is None
    finally:
        torch.use_deterministic_algorithms(False)
