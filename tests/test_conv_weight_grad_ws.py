"""Workspace of the sparse convolution's weight gradient: its size by the path that will run, and the CUDA-core path
with less of it or none.

FP32 sums of m products in any order are within m 2^-24 of the sum of their magnitudes (Higham, first order); a 16-bit
result adds half a unit in its last place.
"""
import pytest
import torch

from jspsr import _lib as L


@pytest.mark.parametrize("K,cin,cout,pairs", [(27, 256, 256, 32768), (27, 64, 64, 1 << 20), (8, 16, 16, 100), (1, 128, 32, 0)])
def test_bytes(K, cin, cout, pairs):
    lib = L.load()
    one = 4 * K * cin * cout
    tensor_cores = one * min(64, max(1, -(-pairs // 2048)))
    assert lib.ngs_conv_weight_grad_ws_bytes(K, cin, cout, pairs) == tensor_cores
    for dt in (L.NGS_F16, L.NGS_BF16):
        assert lib.ngs_conv_weight_grad_ws_bytes_of(K, cin, cout, pairs, dt) == tensor_cores
    for dt, cols in ((L.NGS_F32, cout), (L.NGS_F16, cout + 1)):
        one = 4 * K * cin * cols
        splits, rest = divmod(lib.ngs_conv_weight_grad_ws_bytes_of(K, cin, cols, pairs, dt), one)
        tiles = K * -(-cin // 64) * -(-cols // 64)
        assert rest == 0 and 1 <= splits <= min(64, max(1, -(-pairs // 512)))
        assert (splits - 1) * tiles <= 2400


@pytest.mark.gpu
@pytest.mark.parametrize("cin,cout,dtype", [(16, 32, torch.float32), (70, 65, torch.float32), (8, 20, torch.bfloat16)])
def test_any_workspace(cin, cout, dtype):
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(cin)
    K, n, counts = 3, 500, [5000, 0, 1337]
    x, gy = torch.randn(n, cin, generator=g, device=dev).to(dtype), torch.randn(n, cout, generator=g, device=dev).to(dtype)
    maps = torch.randint(n, (sum(counts), 2), generator=g, device=dev).int()
    starts = torch.tensor([0, 5000, 5000, 6337], device=dev)
    want = torch.zeros(K, cin, cout, dtype=torch.float64, device=dev)
    mag = torch.zeros_like(want)
    for k in range(K):
        i, o = maps[starts[k]:starts[k + 1]].long().T
        want[k], mag[k] = x.double()[i].T @ gy.double()[o], x.double().abs()[i].T @ gy.double().abs()[o]
    dt = {torch.float32: L.NGS_F32, torch.bfloat16: L.NGS_BF16}[dtype]
    one = 4 * K * cin * cout
    full = L.load().ngs_conv_weight_grad_ws_bytes_of(K, cin, cout, max(counts), dt)
    assert full > 3 * one
    for size in (0, one - 4, one, 5 * one // 2, full, full + one):
        ws = torch.empty(size, dtype=torch.uint8, device=dev)
        gw, err = torch.full((K, cin, cout), float("nan"), dtype=dtype, device=dev), torch.zeros(1, dtype=torch.int32, device=dev)
        L.call("ngs_conv_weight_grad", L.ptr(x), n, cin, L.ptr(gy), n, cout, L.ptr(maps), L.ptr(starts), K, max(counts), 0,
               dt, L.ptr(gw), int(dtype == torch.float32), L.ptr(ws) if size else None, size, L.ptr(err), L.stream())
        assert int(err) == 0
        bound = max(counts) * 2.0 ** -24 * mag
        bound = bound + (2.0 ** -8 * (want.abs() + bound) if dtype == torch.bfloat16 else 0)
        assert ((gw.double() - want).abs() <= bound + 1e-30).all()
