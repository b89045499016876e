"""CPU: the order of the backward's work items (ItemOrder in csrc/tile_order.cuh, which the kernels call) gives every (pair, block) exactly one number,
for chunks of one pair, of all pairs and in between."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flash-attention-npu_b200", "csrc")
SOURCE = r"""
#include <cstdio>
#include <set>
#include <utility>
#include "tile_order.cuh"
int main() {
  for (int pairs : {1, 2, 7, 48})
    for (int blocks : {1, 2, 24})
      for (int chunk : {1, 2, 5, pairs}) {
        if (chunk > pairs) continue;
        fa::ItemOrder order;
        order.set(blocks, pairs, chunk);
        std::set<std::pair<int, int>> seen;
        int last_chunk = 0, last_block = 0;
        for (int t = 0; t < pairs * blocks; ++t) {
          const fa::ItemPlace at = order.place(t);
          const int ck = at.pair / chunk;
          if (at.pair < 0 || at.pair >= pairs || at.block < 0 || at.block >= blocks || !seen.insert({at.pair, at.block}).second ||
              ck < last_chunk || (ck == last_chunk && at.block < last_block)) {
            std::printf("pairs %d blocks %d chunk %d item %d: pair %d block %d\n", pairs, blocks, chunk, t, at.pair, at.block);
            return 1;
          }
          last_chunk = ck;
          last_block = at.block;
        }
      }
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_every_work_item_has_one_number(tmp_path):
    src, exe = tmp_path / "items.cpp", tmp_path / "items"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-fsanitize=undefined", "-fno-sanitize-recover", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    subprocess.run([str(exe)], check=True)
