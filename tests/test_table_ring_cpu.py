"""The footprint ring of the pipelined table solve (csrc/ws_ring.cuh) on the CPU: a
model of its loader, producer groups and tensor-core issuer over barriers that
know the parity of a phase only, as mbarriers do, with the box loads completing
in any order.  Whenever a group's wait returns, its tile's footprint is the one
in the buffer, and every tile gets through."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))

MODEL = r"""
#include "ws_ring.cuh"
#include <cstdio>
#include <random>
#include <vector>

struct Bar {  // completed phases; a wait on a parity passes unless the phase under way has it
  int done = 0;
  bool ready(uint32_t parity) const { return (uint32_t)(done & 1) != parity; }
};

template <int BUFS, int GROUPS>
int run(unsigned seed, int tiles) {
  using Ring = arb::FootprintRing<BUFS, GROUPS>;
  std::mt19937 rng(seed);
  std::vector<Bar> full(Ring::FULL), empty(BUFS);
  std::vector<int> holds(BUFS, -1), at(GROUPS), stage(GROUPS, 0), flight;
  std::vector<bool> ready(tiles, false);
  int issued = 0, mma = 0, idle = 0;  // mma: tiles whose products are done, in order
  for (int g = 0; g < GROUPS; ++g) at[g] = g;
  const int slow = (int)(rng() % tiles);  // this tile's load takes long
  auto finished = [&] {
    for (int g = 0; g < GROUPS; ++g)
      if (at[g] < tiles) return false;
    return true;
  };
  while (!finished()) {
    if (++idle > 200000) return 2;  // no tile got through for long: a hand-off is missing
    const unsigned who = rng() % (GROUPS + 3);
    if (who == 0) {  // loader
      if (issued < tiles &&
          (issued < BUFS || empty[Ring::buffer(issued - BUFS)].ready(Ring::empty_parity(issued - BUFS))))
        flight.push_back(issued++);
    } else if (who == 1) {  // some box arrives
      if (!flight.empty()) {
        const size_t i = rng() % flight.size();
        if (flight[i] == slow && rng() % 1000) continue;
        holds[Ring::buffer(flight[i])] = flight[i];
        ++full[Ring::full(flight[i])].done;
        flight.erase(flight.begin() + (long)i);
      }
    } else if (who == 2) {  // tensor-core issuer
      if (mma < tiles && ready[mma]) ++mma;
    } else {  // a producer group
      const int g = (int)who - 3, k = at[g];
      if (k >= tiles) continue;
      if (stage[g] == 0) {
        if (!full[Ring::full(k)].ready(Ring::full_parity(k))) continue;
        if (holds[Ring::buffer(k)] != k) return 1;  // another tile's footprint
        ++empty[Ring::buffer(k)].done;
        stage[g] = 1;
      } else if (k < GROUPS || mma > k - GROUPS) {  // the tile before in this operand buffer is used up
        ready[k] = true;
        stage[g] = 0;
        at[g] += GROUPS;
        idle = 0;
      }
    }
  }
  return 0;
}

int main() {
  for (unsigned seed = 1; seed <= 400; ++seed) {
    const int tiles = 1 + (int)(seed % 37);
    const int r = run<3, 2>(seed, tiles) | run<2, 2>(seed, tiles) << 2 | run<4, 2>(seed, tiles) << 4 |
                  run<3, 1>(seed, tiles) << 6;
    if (r) {
      std::printf("seed %u, %d tiles: %d\n", seed, tiles, r);
      return 1;
    }
  }
  return 0;
}
"""


def test_a_group_only_reads_its_own_tiles(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src = tmp_path / "ring.cpp"
    src.write_text(MODEL)
    exe = tmp_path / "ring"
    subprocess.run([cxx, "-O1", "-std=c++17", "-I", os.path.join(ROOT, "arbinterp_gb300", "csrc"), str(src), "-o",
                    str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
