"""The tensor-core gather GEMM on channels that are no multiple of 16 (a row is an odd number of 16-byte pieces), below,
at and above the number of rows from which a tile has 96 of its rows copied another way.

Products of 16-bit values are exact in FP32; the FP32 sum of m of them is within m 2^-23 of the sum of their
magnitudes (twice the round-to-nearest bound: the tensor core's adds may truncate).
"""
import pytest
import torch

from jspsr import _lib as L

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("kdim,ncols,dtype", [(8, 16, torch.bfloat16), (24, 32, torch.float16), (72, 48, torch.bfloat16),
                                              (136, 272, torch.float16)])
@pytest.mark.parametrize("n_rows", [31, 128 * 148, 128 * 148 + 1, 40_001])
def test_gather_gemm(kdim, ncols, dtype, n_rows):
    g = torch.Generator(device=DEV).manual_seed(n_rows + kdim)
    n_src, K = 700, 5
    x = torch.randn((n_src, kdim), device=DEV, generator=g).to(dtype)
    w = torch.randn((K, ncols, kdim), device=DEV, generator=g).to(dtype)
    table = torch.randint(-n_src // 2, n_src + 20, (K, n_rows), device=DEV, generator=g).int()
    table[K // 2] = -1                                                # an offset no tile has a pair of
    table[:, n_rows // 2:n_rows // 2 + 130] = -1                      # and rows without any
    ref = torch.zeros((n_rows, ncols), dtype=torch.float64, device=DEV)
    mag = torch.zeros_like(ref)
    for k in range(K):
        m = (table[k] >= 0) & (table[k] < n_src)
        rows = x.double()[table[k][m].long()]
        ref[m] += rows @ w[k].double().T
        mag[m] += rows.abs() @ w[k].double().abs().T
    out = torch.full((n_rows, ncols), float("nan"), device=DEV)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    L.call("ngs_conv_gather_gemm_kmajor", L.ptr(x), n_src, kdim, L.ptr(table), n_rows, K, L.ptr(w), ncols,
           L.NGS_BF16 if dtype == torch.bfloat16 else L.NGS_F16, L.ptr(out), 1, L.ptr(err), L.stream())
    assert int(err) == 0
    assert ((out - ref).abs() <= K * kdim * 2.0 ** -23 * mag).all()
