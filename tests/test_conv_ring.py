"""The stage ring of the convolution's tile kernels, run on the host: wherever a producer's walk ends -- at its last step,
or giving up at any wait, the one for the end marker too -- the span it returns holds exactly the copies that nothing
has been waited for, each still the last step of its stage (so that its barrier's parity tells)."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "neural-galerkin_b200" / "csrc"

SOURCE = r"""
#include <cstdio>
#include <vector>
#include "conv_ring.h"
// a line per walk: stages, steps, wait that gives up (-1: none), first, last, in flight..., -1
int main() {
  for (int S = 2; S <= 8; S++)
    for (int T = 0; T <= 3 * S + 1; T++)
      for (int stop = -1; stop <= T; stop++) {
        int at = 0, k = 0;
        std::vector<int> stage_step(S, -1), copies;
        std::vector<char> landed;
        bool wrong = false;
        const RingSpan span = ring_walk(
            S, [&] { return at++ < T ? 64 : 0; },
            [&](int st, uint32_t parity, bool fresh) {
              const int step = at - 1;
              if (fresh != (step < S) || st != step % S) wrong = true;
              if (fresh) return true;
              if (parity != (uint32_t)((step / S - 1) & 1)) wrong = true;
              if (k++ == stop) return false;
              if (stage_step[st] >= 0) landed[stage_step[st]] = 1;
              return true;
            },
            [&](int st, int valid) {
              const int step = at - 1;
              stage_step[st] = step;
              if (valid > 0) { copies.push_back(step); landed.push_back(0); }
            });
        std::printf("%d %d %d %d %d %d", S, T, stop, (int)wrong, span.first, span.last);
        for (size_t i = 0; i < copies.size(); i++)
          if (!landed[i]) std::printf(" %d", stage_step[copies[i] % S] == copies[i] ? copies[i] : -2);
        std::printf("\n");
      }
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_walk_ends_with_the_copies_in_flight(tmp_path):
    src = tmp_path / "ring.cpp"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", f"-I{CSRC}", str(src), "-o", str(tmp_path / "ring")], check=True)
    out = subprocess.run([str(tmp_path / "ring")], check=True, capture_output=True, text=True).stdout
    lines = [[int(v) for v in line.split()] for line in out.splitlines()]
    assert len(lines) > 500
    for S, T, stop, wrong, first, last, *flying in lines:
        assert not wrong
        # the waits of a walk: steps S .. T (T: the marker)
        assert flying == list(range(first, last)), (S, T, stop)
        assert 0 <= first and last <= T and last - first <= S
