"""The CUDA-core tiles of the sparse convolution (FP32 features, and 16-bit channel counts that the tensor
cores do not take) at the edges of their row, column and channel tiles, against the same sums in FP64.

Bounds: FP32 sums of m products in any order are within m * 2^-24 of the sum of their magnitudes
(Higham, first order); a 16-bit result adds half a unit in its last place.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)
ULP = {torch.float32: 0.0, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


def layer(n_in, n_out, K, seed):
    rng = np.random.default_rng(seed)
    pairs, sizes = [], []
    for k in range(K):
        m = 0 if k == 1 else int(rng.integers(0, min(n_in, n_out) + 1))       # one offset without pairs
        pairs.append(np.stack([rng.permutation(n_in)[:m], np.sort(rng.permutation(n_out)[:m])], 1))
        sizes.append(m)
    return torch.from_numpy(np.concatenate(pairs).astype(np.int32)).to(DEV), torch.tensor(sizes, dtype=torch.int32)


@pytest.mark.parametrize("n_in,n_out", [(1, 1), (63, 65), (300, 129), (2000, 1500)])
@pytest.mark.parametrize("cin,cout,dtype", [(1, 1, torch.float32), (4, 16, torch.float32), (16, 17, torch.float32),
                                            (17, 33, torch.float32), (32, 64, torch.float32), (65, 70, torch.float32),
                                            (4, 20, torch.float16), (6, 40, torch.bfloat16)])
def test_forward_and_gradients(n_in, n_out, cin, cout, dtype):
    from jspsr.sparse_conv import sparse_conv
    K = 8
    maps, sizes = layer(n_in, n_out, K, n_in + cin)
    g = torch.Generator(device=DEV).manual_seed(cin * 100 + cout)
    x, w, gy = (torch.randn(*s, generator=g, device=DEV).to(dtype) for s in ((n_in, cin), (K, cin, cout), (n_out, cout)))
    xr, wr = x.clone().requires_grad_(True), w.clone().requires_grad_(True)
    y = sparse_conv(xr, wr, maps, sizes, (n_in, n_out))
    gx, gw = torch.autograd.grad(y, [xr, wr], gy)
    want = [torch.zeros(n_out, cout), torch.zeros(n_in, cin), torch.zeros(K, cin, cout)]
    mags = [t.clone().double() for t in want]
    want = [t.double() for t in want]
    X, W, G = (t.double().cpu() for t in (x, w, gy))
    at = 0
    for k, m in enumerate(sizes.tolist()):
        i, o = maps[at:at + m, 0].long().cpu(), maps[at:at + m, 1].long().cpu()
        at += m
        for sign, out in ((lambda t: t, want), (torch.abs, mags)):
            out[0].index_add_(0, o, sign(X)[i] @ sign(W)[k])
            out[1].index_add_(0, i, sign(G)[o] @ sign(W)[k].T)
            out[2][k] = sign(X)[i].T @ sign(G)[o]
    terms = [K * cin, K * cout, max(1, int(sizes.max()))]
    for got, ref, mag, m in zip((y.detach(), gx, gw), want, mags, terms):
        bound = (m + 2) * 2.0 ** -24 * mag + ULP[dtype] * (ref.abs() + (m + 2) * 2.0 ** -24 * mag) + 1e-30
        assert ((got.double().cpu() - ref).abs() <= bound + (2.0 ** -24 if dtype == torch.float16 else 0.0)).all()


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_non_finite_weights_reach_only_the_rows_with_a_pair(bad):
    """An infinite or NaN weight of one offset touches the outputs that have a pair of that offset, and no other."""
    from jspsr.sparse_conv import sparse_conv
    n, K, cin, cout = 200, 8, 20, 24
    maps, sizes = layer(n, n + 1, K, 5)
    x, w = torch.rand(n, cin, device=DEV) + 0.5, torch.rand(K, cin, cout, device=DEV)
    w[3, 7, 11] = bad
    y = sparse_conv(x, w, maps, sizes, (n, n + 1))
    at = int(sizes[:3].sum())
    hit = torch.zeros(n + 1, dtype=torch.bool, device=DEV)
    hit[maps[at:at + int(sizes[3]), 1].long()] = True
    assert torch.equal(~torch.isfinite(y[:, 11]), hit) and torch.isfinite(y[:, :11]).all() and torch.isfinite(y[:, 12:]).all()


@pytest.mark.parametrize("n_in,n_out", [(70, 127), (300, 128), (513, 400)])
@pytest.mark.parametrize("cin,cout,dtype", [(16, 24, torch.float32), (64, 64, torch.float16), (40, 272, torch.bfloat16)])
def test_both_table_layouts_give_the_same_bits(n_in, n_out, cin, cout, dtype):
    """Tables with the row outermost (ngs_conv_table) and with the offset outermost (.._kmajor)."""
    from jspsr import _lib as L, ext
    K = 8
    maps, sizes = layer(n_in, n_out, K, n_out)
    starts, _ = ext._offset_starts(sizes, K, DEV)
    x, w = torch.randn(n_in, cin, device=DEV).to(dtype), torch.randn(K, cout, cin, device=DEV).to(dtype)
    y = [torch.empty(n_out, cout, device=DEV, dtype=dtype) for _ in range(2)]
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    tables = [torch.empty(n_out, K, dtype=torch.int32, device=DEV), torch.empty(K, n_out, dtype=torch.int32, device=DEV)]
    for t, out, end in zip(tables, y, ("", "_kmajor")):
        L.call("ngs_conv_table" + end, L.ptr(maps), L.ptr(starts), K, 1, n_out, -1, L.ptr(t), L.stream())
        L.call("ngs_conv_gather_gemm" + end, L.ptr(x), n_in, cin, L.ptr(t), n_out, K, L.ptr(w), cout, ext._conv_dtype(x),
               L.ptr(out), int(dtype == torch.float32), L.ptr(err), L.stream())
    assert torch.equal(tables[0].T, tables[1]) and torch.equal(y[0], y[1]) and int(err) == 0
