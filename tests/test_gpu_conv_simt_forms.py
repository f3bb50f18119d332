"""The two forms of the CUDA-core gather GEMM, tiles and a thread per output: the first rows of a layer that runs in
tiles, computed as a small layer of their own by a thread per output, come out the same bit for bit (both add a row's
products in one order), with missing and out-of-range rows and with weights that are not finite; and both are right.

FP32 sums of m products are within m 2^-24 of the sum of their magnitudes (Higham, first order); a 16-bit result adds
half a unit in its last place.
"""
import shutil
import subprocess
from pathlib import Path

import pytest
import torch

from jspsr import _lib as L

CSRC = Path(__file__).resolve().parents[1] / "neural-galerkin_b200" / "csrc"
# channels in and out, type, rows of the small layer
LAYERS = [(16, 16, torch.float32, 700), (16, 33, torch.float32, 100), (4, 64, torch.float32, 129), (7, 20, torch.float32, 65),
          (64, 4, torch.float32, 1000), (65, 70, torch.float32, 1), (144, 12, torch.bfloat16, 63), (6, 256, torch.float16, 64)]


@pytest.fixture(scope="module")
def by_thread(tmp_path_factory):
    """Rows, channels in and out, bytes of an element -> whether the layer runs by thread."""
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    where = tmp_path_factory.mktemp("plan")
    (where / "plan.cpp").write_text("""
#include <cstdio>
#include <cstdlib>
#include "conv_plan.h"
int main(int, char** v) {
  std::printf("%d", (int)conv::simt_by_thread(std::atoll(v[1]), std::atoi(v[2]), std::atoi(v[3]), std::atoi(v[4])));
}
""")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", f"-I{CSRC}", "plan.cpp", "-o", "plan"], cwd=where, check=True)
    return lambda *a: bool(int(subprocess.run([str(where / "plan"), *map(str, a)], capture_output=True, check=True).stdout))


def test_rule(by_thread):
    # one line: a layer that runs by thread does so with fewer rows, too
    for cin, cout, size in ((4, 16, 4), (16, 16, 4), (48, 32, 4), (256, 4, 4), (144, 4, 2), (6, 256, 2)):
        runs = [by_thread(rows, cin, cout, size) for rows in (1, 300, 3000, 30000, 300000, 1 << 31)]
        assert runs == sorted(runs, reverse=True) and not runs[-1]
    assert by_thread(3000, 4, 16, 4) and not by_thread(30000, 16, 32, 4)


def rows_of(by_thread, cin, cout, size):
    """Rows (not a multiple of a tile's) of a layer that runs in tiles: twice what the rule asks for, or less."""
    return next(r for r in (1001 << k for k in range(12)) if not by_thread(r, cin, cout, size)) | 1


def test_layers(by_thread):
    for cin, cout, dtype, small in LAYERS:
        size = torch.finfo(dtype).bits // 8
        assert by_thread(small, cin, cout, size) and rows_of(by_thread, cin, cout, size) < 1 << 19


@pytest.mark.gpu
@pytest.mark.parametrize("cin,cout,dtype,small", LAYERS)
@pytest.mark.parametrize("bad", [None, float("inf"), float("nan")])
def test_forms_agree(cin, cout, dtype, small, bad, by_thread):
    dev = torch.device("cuda", 0)
    rows = rows_of(by_thread, cin, cout, torch.finfo(dtype).bits // 8)
    g = torch.Generator(device=dev).manual_seed(cin + cout)
    K, n_src = 5, 400
    x, w = torch.randn(n_src, cin, generator=g, device=dev).to(dtype), torch.randn(K, cout, cin, generator=g, device=dev).to(dtype)
    if bad is not None:
        w[2, cout // 2, cin // 2] = bad
    table = torch.randint(-n_src // 2, n_src + 20, (K, rows), generator=g, device=dev).int()
    table[1] = -1                                              # an offset without a pair
    outs = []
    for m in (rows, small):
        for name, t in (("ngs_conv_gather_gemm_kmajor", table[:, :m].contiguous()), ("ngs_conv_gather_gemm", table[:, :m].T.contiguous())):
            out, err = torch.full((m, cout), 7.0, dtype=dtype, device=dev), torch.zeros(1, dtype=torch.int32, device=dev)
            L.call(name, L.ptr(x), n_src, cin, L.ptr(t), m, K, L.ptr(w), cout,
                   {torch.float32: L.NGS_F32, torch.bfloat16: L.NGS_BF16, torch.float16: L.NGS_F16}[dtype], L.ptr(out),
                   int(dtype == torch.float32), L.ptr(err), L.stream())
            assert int(err) == 0
            outs.append(out)
    for o in outs[1:]:
        a = outs[0][:len(o)]
        assert torch.equal(torch.isnan(o), torch.isnan(a)) and torch.equal(torch.nan_to_num(o), torch.nan_to_num(a))
    if bad is None:
        ref = torch.zeros(rows, cout, dtype=torch.float64, device=dev)
        mag = torch.zeros_like(ref)
        for k in range(K):
            m = (table[k] >= 0) & (table[k] < n_src)
            src = x.double()[table[k][m].long()]
            ref[m] += src @ w[k].double().T
            mag[m] += src.abs() @ w[k].double().abs().T
        bound = K * cin * 2.0 ** -24 * mag
        bound = bound + {torch.float32: 0.0, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}[dtype] * (ref.abs() + bound)
        assert ((outs[0].double() - ref).abs() <= bound + 2.0 ** -24 * (dtype == torch.float16)).all()
