"""Plan of the gather GEMM's blocks for every tile width: what an SM is planned to hold fits its tensor memory (a block
allocates a power of two of columns) and its shared memory, and a block gets all the stages that its share has room for."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "neural-galerkin_b200" / "csrc"

SOURCE = r"""
#include <cstdio>
#include "conv_plan.h"
int main() {
  for (int box = 16; box <= 256; box += 16) {
    const conv::GatherPlan p = conv::gather_plan(box);
    std::printf("%d %d %d %u %zu %u\n", box, p.per_sm, p.stages, p.stage_bytes, p.smem, conv::tmem_columns(box));
  }
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_planned_blocks_fit_an_sm(tmp_path):
    src = tmp_path / "plan.cpp"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", f"-I{CSRC}", str(src), "-o", str(tmp_path / "plan")], check=True)
    out = subprocess.run([str(tmp_path / "plan")], check=True, capture_output=True, text=True).stdout
    plans = [[int(v) for v in line.split()] for line in out.splitlines()]
    assert [p[0] for p in plans] == list(range(16, 257, 16))
    for box, per_sm, stages, stage_bytes, smem, columns in plans:
        assert columns >= max(box, 32) and columns & (columns - 1) == 0
        assert per_sm >= 1 and per_sm * columns <= 512
        assert stage_bytes >= (128 + box) * 128 and stage_bytes % 1024 == 0
        assert 2 <= stages <= 8
        # 1.5 KB of a block are its static arrays and the SM's reserve
        assert smem == 1024 + stages * stage_bytes and per_sm * (smem + 1536) <= 227 << 10
        assert stages == 8 or per_sm * (smem + stage_bytes + 1536) > 227 << 10
