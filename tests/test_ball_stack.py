"""The radius balls' shared stacks hold every walk, whatever the tree.

A ball's walk takes as many nodes off its stack as segment.cuh's ball_width says and puts up to two
back for each. This plays that rule against trees as deep as a Karras tree over 63-bit codes and
32-bit indices can be (95 nodes on a path), the whole tree within the ball: no walk may need more
entries than its kernel has.
"""

from __future__ import annotations

import subprocess
from importlib import import_module

HARNESS = r"""
#include "segment.cuh"
#include <cstdio>
#include <random>
using namespace sherd;

int most(uint32_t stack, int threads, int shape) {
  std::mt19937 rng(shape);
  std::vector<int> level{1};  // of the nodes waiting, the root on level 1
  size_t most = 1;
  for (int step = 0; step < 200000 && !level.empty(); ++step) {
    const int width = ball_width(int(level.size()), stack, threads);
    if (width < 1 || width > int(level.size()) || width > threads) return -1;
    const std::vector<int> taken(level.end() - width, level.end());
    level.resize(level.size() - width);
    for (int child = 0; child < 2; ++child)
      for (int l : taken)
        if (l < 95 && (child == 0 || shape == 0 || rng() % 16 >= unsigned(shape))) level.push_back(l + 1);
    most = std::max(most, level.size());
  }
  return int(most);
}

int main() {
  for (int shape = 0; shape < 16; ++shape)
    std::printf("%d %u %d %u\n", most(BALL_STACK, 32, shape), BALL_STACK,
                most(BALL_BLOCK_STACK, BALL_BLOCK, shape), BALL_BLOCK_STACK);
}
"""


def test_no_walk_outgrows_its_stack(tmp_path):
    build = import_module("sherd-refit_b200.build")
    src, exe = tmp_path / "stack.cu", tmp_path / "stack"
    src.write_text(HARNESS)
    flags = [f for f in build.FLAGS if f not in ("-Xptxas", "-v", "-shared", "-lineinfo")]
    subprocess.run([build.NVCC, *flags, "-I", str(build.SRC), str(src), "-o", str(exe)], check=True,
                   capture_output=True)
    rows = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")
    rows = [[int(x) for x in r.split()] for r in rows if r]
    assert len(rows) == 16
    for warp, warp_stack, block, block_stack in rows:
        assert 0 < warp <= warp_stack and 0 < block <= block_stack, rows
