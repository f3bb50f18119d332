"""The tensor-core gather GEMM at the edges of its tiles (128 rows, 64 channels a step, 256 columns, one offset or the
most), with missing and out-of-range table entries, offsets without a pair, and both orders of the table.

Products of 16-bit values are exact in FP32; the FP32 sum of m of them is within m 2^-23 of the sum of their
magnitudes (twice the round-to-nearest bound: the tensor core's adds may truncate).
"""
import pytest
import torch

from jspsr import _lib as L

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n_rows,n_src,kdim,ncols,K", [
    (1, 1, 8, 16, 1), (127, 40, 64, 64, 27), (128, 300, 72, 48, 3), (129, 129, 64, 256, 27), (300, 0, 64, 64, 4),
    (1000, 700, 136, 272, 2), (515, 515, 24, 32, 125), (2500, 2000, 128, 128, 8)])
def test_gather_gemm(dtype, n_rows, n_src, kdim, ncols, K):
    g = torch.Generator(device=DEV).manual_seed(n_rows + kdim)
    x = torch.randn((n_src, kdim), device=DEV, generator=g).to(dtype)
    w = torch.randn((K, ncols, kdim), device=DEV, generator=g).to(dtype)
    table = torch.randint(-max(n_src, 1), n_src + 20, (K, n_rows), device=DEV, generator=g).int()
    table[K // 2] = -1                                                # an offset no tile has a pair of
    table[:, n_rows // 2:n_rows // 2 + 130] = -1                      # and rows without any
    ref = torch.zeros((n_rows, ncols), dtype=torch.float64, device=DEV)
    mag = torch.zeros_like(ref)
    for k in range(K):
        m = (table[k] >= 0) & (table[k] < n_src)
        rows = x.double()[table[k][m].long()]
        ref[m] += rows @ w[k].double().T
        mag[m] += rows.abs() @ w[k].double().abs().T
    outs = []
    for name, t in (("ngs_conv_gather_gemm_kmajor", table), ("ngs_conv_gather_gemm", table.T.contiguous())):
        out = torch.full((n_rows, ncols), float("nan"), device=DEV)
        err = torch.zeros(1, dtype=torch.int32, device=DEV)
        L.call(name, L.ptr(x), n_src, kdim, L.ptr(t), n_rows, K, L.ptr(w), ncols,
               L.NGS_BF16 if dtype == torch.bfloat16 else L.NGS_F16, L.ptr(out), 1, L.ptr(err), L.stream())
        assert int(err) == 0
        assert ((out - ref).abs() <= K * kdim * 2.0 ** -23 * mag).all()
        outs.append(out)
    assert torch.equal(*outs)
