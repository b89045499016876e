"""CPU: the order of the query tiles of ragged input (csrc/tile_order.cuh, the arithmetic of the prefill kernel's run-time tile
draw) gives every tile exactly one position, whichever order the positions are asked for in."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flash-attention-npu_b200", "csrc")
SOURCE = r"""
#include <algorithm>
#include <cstdio>
#include <random>
#include <set>
#include <tuple>
#include <vector>
#include "tile_order.cuh"
struct Levels {
  std::vector<int> lo, n;
  int live = 0, top = 0;
  int count(int level) const {
    int c = 0;
    for (size_t i = 0; i < lo.size(); ++i) c += level >= lo[i] && level < lo[i] + n[i];
    return c;
  }
};
int main() {
  std::mt19937 rng(7);
  auto pick = [&](int lo, int hi) { return lo + (int)(rng() % (unsigned)(hi - lo + 1)); };
  for (int round = 0; round < 600; ++round) {
    Levels lv;
    const int b = pick(1, 70), heads = pick(1, 9), chunk = round % 3 ? pick(1, heads) : heads;
    for (int i = 0; i < b; ++i) {
      lv.lo.push_back(pick(0, 3) ? pick(0, 12) : 0);
      lv.n.push_back(pick(0, 4) ? pick(1, 6) : 0);
      lv.live += lv.n[i];
      if (lv.n[i]) lv.top = std::max(lv.top, lv.lo[i] + lv.n[i] - 1);
    }
    std::vector<int> order;
    for (int i = 0; i < lv.live * heads + 5; ++i) order.push_back(i);
    if (round % 4 == 1) std::reverse(order.begin(), order.end());
    if (round % 4 == 2) std::shuffle(order.begin(), order.end(), rng);
    if (round % 4 == 3)  // growing, with neighbours exchanged now and then
      for (size_t i = 0; i + 1 < order.size(); i += pick(1, 6)) std::swap(order[i], order[i + 1]);
    fa::TileCursor cur;
    std::set<std::tuple<int, int, int>> seen;  // (batch entry, head, tile)
    for (int n : order) {
      int head, rank;
      const bool got = fa::tile_locate(cur, lv, heads, chunk, n, head, rank);
      if (got != (n < lv.live * heads)) { std::printf("position %d of %d: %d\n", n, lv.live * heads, got); return 1; }
      if (!got) continue;
      int bi = -1;
      for (int i = 0, r = rank; i < b; ++i)
        if (cur.level >= lv.lo[i] && cur.level < lv.lo[i] + lv.n[i] && r-- == 0) bi = i;
      if (rank < 0 || bi < 0 || head < 0 || head >= heads) { std::printf("position %d: head %d rank %d\n", n, head, rank); return 1; }
      if (head / chunk != n / (lv.live * chunk)) { std::printf("position %d: head %d outside its chunk\n", n, head); return 1; }
      if (!seen.insert({bi, head, cur.level - lv.lo[bi]}).second) { std::printf("position %d: a tile twice\n", n); return 1; }
    }
    if ((int)seen.size() != lv.live * heads) { std::printf("%zu tiles of %d\n", seen.size(), lv.live * heads); return 1; }
  }
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_every_tile_has_one_position_in_any_order(tmp_path):
    src, exe = tmp_path / "order.cpp", tmp_path / "order"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-fsanitize=undefined", "-fno-sanitize-recover", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


DIVISION = r"""
#include <cstdio>
#include <random>
#include "tile_order.cuh"
int main() {
  std::mt19937 rng(3);
  std::uniform_int_distribution<int> any(0, 0x7fffffff);
  for (int k = 0; k < 4000; ++k) {
    const int d = k < 2000 ? k + 1 : k < 2060 ? (k % 2 ? (1 << (k - 2000) / 2) : 0x7fffffff - (k - 2000)) : any(rng) >> (k % 31);
    fa::FastDiv f;
    f.set(d);
    if (d < 1) continue;
    for (int i = 0; i < 400; ++i) {
      long long n = i < 4 ? i : i < 8 ? 0x7fffffffLL - (i - 4) : (long long)d * (any(rng) / d) + (i % 3) - 1;
      if (n < 0 || n > 0x7fffffffLL) n = any(rng);
      if (f.div((int)n) != (int)n / d) { std::printf("%lld / %d: %d\n", n, d, f.div((int)n)); return 1; }
    }
  }
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_division_by_multiplication(tmp_path):
    """Every divisor up to 2000, powers of two, the largest and random ones; dividends at multiples and one beside them."""
    src, exe = tmp_path / "div.cpp", tmp_path / "div"
    src.write_text(DIVISION)
    subprocess.run(["g++", "-O1", "-std=c++17", "-fsanitize=undefined", "-fno-sanitize-recover", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
