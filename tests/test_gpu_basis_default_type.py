"""Values of an additive basis and their coefficient gradient come in the inputs' type, whatever torch's default
type is."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("default", [torch.float32, torch.float64])
@pytest.mark.parametrize("n", [1, 1000])
def test_values_and_gradient_follow_the_inputs(default, n):
    from jspsr.bases.additive import AdditiveBasis
    from jspsr.bases.additive_components import Bezier, Power
    g = torch.Generator().manual_seed(n)
    comps = [Bezier(), Power(0), Power(1), Power(2), Power(3)]
    basis = AdditiveBasis(comps, [1.0] + [0.0] * 4)
    coef = torch.randn(50, 3 * len(comps), generator=g)
    x = torch.rand(n, 3, generator=g) * 3 - 1.5
    ids = torch.randint(50, (n,), generator=g)
    up = torch.randn(n, generator=g)
    before = torch.get_default_dtype()
    torch.set_default_dtype(default)
    try:
        feat = coef.to(DEV).requires_grad_(True)
        out = basis.evaluate(feat, x.to(DEV), ids.to(DEV))
        grad, = torch.autograd.grad(out, feat, up.to(DEV))
    finally:
        torch.set_default_dtype(before)
    assert out.dtype == grad.dtype == torch.float32
    # the same in 64 bits on the CPU
    c64 = coef.double().requires_grad_(True)
    q = [comp.evaluate(x.double()) for comp in comps]
    axes = sum(qk * c64[ids][:, 3 * k:3 * k + 3] for k, qk in enumerate(q))
    want = axes.prod(1)
    grad64, = torch.autograd.grad(want, c64, up.double())
    # FP32: an axis is a sum of C products, each value of a component within four roundings of max(|q|, 1); the value
    # is a product of three axes, a gradient entry the sum over a row's queries of two axes, a component and `up`
    C, eps = len(comps), 2.0 ** -23
    size = sum(qk.abs().clamp(min=1) * coef.double()[ids][:, 3 * k:3 * k + 3].abs() for k, qk in enumerate(q))
    assert bool(((out.cpu().double() - want).abs() <= 3 * (C + 4) * eps * size.prod(1)).all())
    top = torch.stack([qk.abs().clamp(min=1).amax(1) for qk in q]).amax(0)
    most = torch.zeros(50, dtype=torch.float64).index_add_(0, ids, up.double().abs() * top * size.amax(1) ** 2)
    terms = torch.bincount(ids, minlength=50).double()
    assert bool(((grad.cpu().double() - grad64).abs() <= ((2 * (C + 4) + 4 + terms) * eps * most)[:, None] + 1e-30).all())
