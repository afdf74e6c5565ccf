"""The lockstep decision's launch plan (csrc/launch_plan.h), on the CPU: for every size, grid and block the claims cover
the arenas, and a call whose arenas fit the grid in one round gives no warp a second claim (a warp steps its claims one
after another, a whole decision each)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "rocketsim-cuda_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <initializer_list>
#include "launch_plan.h"
using namespace rsx;
int main() {
  long plans = 0, one_round = 0, narrow = 0, bad = 0;
  const uint32_t grids[] = {1, 3, 37, 148, 149, 296, 592, 1480};
  for (uint32_t grid : grids)
    for (uint32_t block = 32; block <= 512; block += 32)
      for (uint32_t split : {0u, 7u, 14u, 15u})
        for (uint64_t k = 1; k <= 3u * grid * block; k += 1 + k / 40) {
          const uint32_t n = (uint32_t)k;
          const LockstepPlan p = lockstep_plan(n, grid, block, split);
          const uint32_t claims = (n + p.width - 1) / p.width;
          const bool one = n <= (uint64_t)grid * block;
          ++plans;
          one_round += one;
          narrow += p.width < 32;
          bool ok = p.width >= 1 && p.width <= 32 && p.block >= 32 && p.block <= block && p.block % 32 == 0 && p.queue == !one &&
                    (split == kSpreadSplit || p.block == block);
          if (one) ok = ok && (claims + grid - 1) / grid <= p.block / 32;  // the blocks' shares differ by one claim at most
          if (!ok && bad++ < 5) std::printf("n %u grid %u block %u split %u: block %u width %u queue %d\n", n, grid, block, split, p.block, p.width, p.queue);
        }
  std::printf("plans %ld one-round %ld narrow %ld bad %ld\n", plans, one_round, narrow, bad);
  return bad != 0;
}
"""


def test_one_round_gives_no_warp_two_claims(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "plan.cpp", tmp_path / "plan"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", CSRC, str(src), "-o", str(exe)], check=True, capture_output=True, text=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout
    words = out.stdout.split()
    for name in ("one-round", "narrow"):
        assert int(words[words.index(name) + 1]) > 1000, out.stdout
