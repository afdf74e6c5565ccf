"""The lockstep decision's launch plan (csrc/launch_plan.h), on the CPU, over sizes, grids and blocks: a call whose arenas
fit the grid in one round gives no warp a second claim (a warp steps its claims one after another, a whole decision each),
and a grid past the SMs is launched with no more blocks than the device holds at once and, below that, no more than hold
the arenas."""
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
  // the grid on 148 SMs that hold `held` blocks each
  long capped = 0;
  for (uint32_t grid : {1u, 37u, 148u, 149u, 296u, 592u, 1480u, 65535u})
    for (uint32_t block = 32; block <= 512; block += 32)
      for (uint32_t held = 1; held <= 8; ++held)
        for (uint64_t k = 1; k <= 400000; k += 1 + k / 10) {
          const uint32_t n = (uint32_t)k, got = lockstep_grid(n, grid, block, 148, [&] { return held; });
          const uint64_t full = 148u * held, lanes = (uint64_t)got * block;
          ++plans;
          capped += got < grid;
          bool ok = got >= 1 && got <= grid && (grid <= 148 ? got == grid : got <= full);
          // fewer blocks than asked for: as many as the device holds, or as many as take the arenas in one round and no SM's worth more
          if (got < grid) ok = ok && got % 148 == 0 && (got == full || (lanes >= n && (got == 148 || lanes - 148ull * block < n)));
          if (!ok && bad++ < 5) std::printf("n %u grid %u block %u held %u: grid %u\n", n, grid, block, held, got);
        }
  std::printf("plans %ld one-round %ld narrow %ld capped %ld bad %ld\n", plans, one_round, narrow, capped, bad);
  return bad != 0;
}
"""


def test_plan(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "plan.cpp", tmp_path / "plan"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", CSRC, str(src), "-o", str(exe)], check=True, capture_output=True, text=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout
    words = out.stdout.split()
    for name in ("one-round", "narrow", "capped"):
        assert int(words[words.index(name) + 1]) > 1000, out.stdout
