"""The barrier word of the 2D relabel and cut (csrc/jfc_flagbar.h): in every order of
arrivals and polls of its blocks, all of them leave behind the same phase, the
first at which none asked for another, and none waits for a block that left."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG

MODEL = r"""
#include <array>
#include <cstdio>
#include <cstdlib>
#include <set>
#include <tuple>
#include <vector>
#include "jfc_flagbar.h"
using jfc::FlagBar;

// asks[block][barrier]; a block arrives, polls until the barrier is complete, and
// goes on if any block asked.  State: per block {barrier, arrived, mine, left}.
struct Block {
  unsigned b = 0, arrived = 0, mine = 0, left = 0;
  bool operator<(const Block& o) const {
    return std::tie(b, arrived, mine, left) < std::tie(o.b, o.arrived, o.mine, o.left);
  }
};
using State = std::pair<unsigned long long, std::vector<Block>>;

int main(int argc, char** argv) {
  const unsigned blocks = (unsigned)atoi(argv[1]), barriers = (unsigned)atoi(argv[2]);
  for (unsigned pattern = 0; pattern < 1u << (blocks * barriers); ++pattern) {
    auto ask = [&](unsigned k, unsigned b) { return b < barriers && (pattern >> (k * barriers + b) & 1u); };
    unsigned last = 0;   // the barrier behind which all leave
    auto any = [&](unsigned b) { bool a = false; for (unsigned k = 0; k < blocks; ++k) a |= ask(k, b); return a; };
    while (any(last)) ++last;
    std::set<State> seen;
    std::vector<State> todo{{0ull, std::vector<Block>(blocks)}};
    while (!todo.empty()) {
      const State st = todo.back();
      todo.pop_back();
      if (!seen.insert(st).second) continue;
      bool moved = false, all_left = true;
      for (unsigned k = 0; k < blocks; ++k) {
        State n = st;
        Block& c = n.second[k];
        if (c.left) continue;
        all_left = false;
        if (!c.arrived) {
          n.first += FlagBar::arrival(c.b, ask(k, c.b), c.mine);
          c.arrived = 1;
        } else {
          if (!FlagBar::complete(n.first, c.b, blocks)) continue;
          const bool more = FlagBar::asked(n.first, c.b);
          if (more != any(c.b)) { printf("pattern %u: block %u misreads barrier %u\n", pattern, k, c.b); return 1; }
          c.arrived = 0;
          if (more) ++c.b;
          else c.left = 1;
        }
        moved = true;
        todo.push_back(n);
      }
      if (!moved && !all_left) { printf("pattern %u: stuck\n", pattern); return 1; }
      if (all_left)
        for (const Block& c : st.second)
          if (c.b != last) { printf("pattern %u: left behind barrier %u, not %u\n", pattern, c.b, last); return 1; }
    }
  }
  // a full grid, every block asking at every barrier, then none
  unsigned long long word = 0;
  std::vector<unsigned> mine(jfc::kFlagBarBlocks, 0u);
  for (unsigned b = 0; b < 40; ++b) {
    for (unsigned k = 0; k < jfc::kFlagBarBlocks; ++k) {
      if (FlagBar::complete(word, b, jfc::kFlagBarBlocks)) { printf("complete too early\n"); return 1; }
      word += FlagBar::arrival(b, b < 37, mine[k]);
    }
    if (!FlagBar::complete(word, b, jfc::kFlagBarBlocks) || FlagBar::asked(word, b) != (b < 37)) {
      printf("full grid: barrier %u misread\n", b);
      return 1;
    }
  }
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_every_order_of_arrivals_and_polls(tmp_path):
    src, exe = tmp_path / "model.cpp", tmp_path / "model"
    src.write_text(MODEL)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(PKG, "csrc"), str(src), "-o", str(exe)], check=True)
    for blocks, barriers in ((1, 3), (2, 4), (3, 3)):
        r = subprocess.run([str(exe), str(blocks), str(barriers)], capture_output=True, text=True)
        assert r.returncode == 0, (blocks, barriers, r.stdout)
