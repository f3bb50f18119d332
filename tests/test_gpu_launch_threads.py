"""Threads that launch one kernel with different amounts of shared memory: none lowers the limit under another's launch
(a launch above the kernel's limit is refused by the host).  The threads are native ones, whose calls overlap."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import pytest
import torch

from jspsr import _lib as L

ROOT = Path(__file__).resolve().parents[1]
pytestmark = [pytest.mark.gpu, pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")]
DEV = torch.device("cuda", 0)
LOOPS = 4000

SOURCE = r"""
#include <atomic>
#include <thread>
#include <cstddef>
#include "ngs.h"
// every entry: the same call from two threads, each on its own stream; the first error, or 0
template <typename F>
static int together(F call, int loops) {
  std::atomic<int> error{0};
  auto run = [&](int which) {
    for (int k = 0; k < loops && !error; k++) {
      const int rc = call(which);
      if (rc) error = rc;
    }
  };
  std::thread other([&] { run(1); });
  run(0);
  other.join();
  return error;
}
extern "C" int pairs(const ngs_basis_pair_term* a, const ngs_basis_pair_term* b, ngs_stream s, ngs_stream t, int loops) {
  return together([&](int w) { return ngs_basis_pairs(w ? b : a, 1, w ? t : s); }, loops);
}
extern "C" int gather(int na, int nb, const void* x, const int32_t* table, const void* bt, void* oa, void* ob, int* err,
                      ngs_stream s, ngs_stream t, int loops) {
  return together([&](int w) {
    return ngs_conv_gather_gemm_kmajor(x, 8, 64, table, 8, 1, bt, w ? nb : na, NGS_BF16, w ? ob : oa, 1, err, w ? t : s);
  }, loops);
}
extern "C" int weight_grad(int na, int nb, const void* x, const void* gy, const int32_t* maps, const int64_t* starts,
                           void* oa, void* ob, void* wa, void* wb, size_t bytes, int* err, ngs_stream s, ngs_stream t,
                           int loops) {
  return together([&](int w) {
    return ngs_conv_weight_grad(x, 8, 64, gy, 8, w ? nb : na, maps, starts, 1, 8, 0, NGS_BF16, w ? ob : oa, 1,
                                w ? wb : wa, bytes, err, w ? t : s);
  }, loops);
}
extern "C" int correction(int na, int nb, const ngs_grid* g, const int32_t* fine, const float* x, const double* tab,
                          double* ra, double* rb, ngs_stream s, ngs_stream t, int loops) {
  return together([&](int w) {
    return ngs_correction_stiffness(fine, 1, 1, *g, x, tab, tab, w ? nb : na, w ? rb : ra, w ? t : s);
  }, loops);
}
"""


@pytest.fixture(scope="module")
def native(tmp_path_factory):
    L.load()
    where = tmp_path_factory.mktemp("threads")
    (where / "threads.cpp").write_text(SOURCE)
    lib = Path(L.__file__).resolve().parent / "libngs.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-pthread", f"-I{ROOT / 'include'}", "threads.cpp",
                    str(lib), "-o", "threads.so"], cwd=where, check=True)
    return C.CDLL(str(where / "threads.so"))


def streams():
    """Two streams whose work comes after everything queued so far."""
    torch.cuda.synchronize()
    made = [torch.cuda.Stream(DEV) for _ in range(2)]
    return made, [C.c_void_p(s.cuda_stream) for s in made]


def test_pair_terms(native):
    """Tables of 10 and of 100 entries, of 12 components: 48 and 150 KB."""
    n, keep, terms = 12, [], []
    for R in (10, 100):
        ff, cs = torch.rand(n, n, R, device=DEV), torch.rand(1, 3 * n, device=DEV)
        ids, rel = torch.zeros(1, dtype=torch.int64, device=DEV), torch.zeros(1, 3, device=DEV)
        one, gs = torch.ones(1, dtype=torch.float64, device=DEV), torch.zeros(1, 3 * n, device=DEV)
        t = L.BasisPairTerm()
        t.ff, t.dd, t.cs, t.ct = ff.data_ptr(), ff.data_ptr(), cs.data_ptr(), cs.data_ptr()
        t.sid, t.tid, t.rel, t.pairs = ids.data_ptr(), ids.data_ptr(), rel.data_ptr(), 1
        t.fscale, t.dscale, t.add, t.C, t.R = 1.0, 1.0, 1.0, n, R
        t.lam, t.xs, t.gs = one.data_ptr(), one.data_ptr(), gs.data_ptr()
        keep.append((ff, cs, ids, rel, one, gs))
        terms.append(t)
    made, raw = streams()
    assert native.pairs(C.byref(terms[0]), C.byref(terms[1]), *raw, LOOPS) == 0
    torch.cuda.synchronize()


def test_convolution(native):
    """16 and 256 output columns, forward and weight gradient."""
    x, gy = (torch.zeros(8, c, dtype=torch.bfloat16, device=DEV) for c in (64, 256))
    w, table = torch.zeros(256, 64, dtype=torch.bfloat16, device=DEV), torch.zeros(1, 8, dtype=torch.int32, device=DEV)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    maps, starts = torch.zeros(8, 2, dtype=torch.int32, device=DEV), torch.tensor([0, 8], device=DEV)
    out = [torch.empty(64, 256, device=DEV) for _ in range(2)]
    ws = [torch.empty(L.load().ngs_conv_weight_grad_ws_bytes(1, 64, 256, 8), dtype=torch.uint8, device=DEV) for _ in range(2)]
    made, raw = streams()
    assert native.gather(16, 256, L.ptr(x), L.ptr(table), L.ptr(w), *map(L.ptr, out), L.ptr(err), *raw, LOOPS) == 0
    assert native.weight_grad(16, 256, L.ptr(x), L.ptr(gy), L.ptr(maps), L.ptr(starts), *map(L.ptr, out), *map(L.ptr, ws),
                              C.c_size_t(ws[0].numel()), L.ptr(err), *raw, LOOPS) == 0
    torch.cuda.synchronize()
    assert int(err) == 0


def test_correction(native):
    """Tables of 3,200 and of 12,000 entries: 50 and 188 KB; a coarse level without voxels."""
    fine = torch.zeros(1, 3, dtype=torch.int32, device=DEV)
    g, words = L.make_grid([0, 0, 0], [1, 1, 1], 2, DEV)
    tab = torch.rand(12000, dtype=torch.float64, device=DEV)
    x, rhs = torch.ones(1, device=DEV), [torch.zeros(1, dtype=torch.float64, device=DEV) for _ in range(2)]
    made, raw = streams()
    assert native.correction(3200, 12000, C.byref(g), L.ptr(fine), L.ptr(x), L.ptr(tab), *map(L.ptr, rhs), *raw, LOOPS) == 0
    torch.cuda.synchronize()
