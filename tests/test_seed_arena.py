"""Host memory of the seed sets (engine.h SeedArena): a replay copies every recursion level's set into its parent's, so a
window whose seeds split off one by one builds D sets of up to D seeds.  The arena's blocks hold the nodes alive at a
time, not every node ever taken, and go between pairs but for the first."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <new>
static size_t held = 0, peak = 0;
void *operator new(size_t n) {
  char *p = static_cast<char *>(std::malloc(n + 16));
  *reinterpret_cast<size_t *>(p) = n;
  held += n;
  if (held > peak) peak = held;
  return p + 16;
}
void operator delete(void *p) noexcept {
  if (!p) return;
  char *q = static_cast<char *>(p) - 16;
  held -= *reinterpret_cast<size_t *>(q);
  std::free(q);
}
void operator delete(void *p, size_t) noexcept { operator delete(p); }
#include "engine.h"
using namespace dcns;
// a chain: each level's seed, then the seeds of the level below, in their order
static void level(int d, int depth, SeedSet &out) {
  out.insert(Seed4{40 * d, 40 * d + 30, 8 * d, 8 * d + 30});
  if (d + 1 == depth) return;
  SeedSet sub;
  level(d + 1, depth, sub);
  for (const Seed4 &s : sub) out.insert(s);
}
int main(int, char **argv) {
  const int depth = std::atoi(argv[1]), windows = std::atoi(argv[2]);
  size_t seeds = 0;
  {
    SeedSet all;
    for (int k = 0; k < windows; ++k) {
      SeedSet one;
      level(0, depth, one);
      seeds += one.size();
      all.insert(one.begin(), one.end());
    }
    seeds += all.size();
  }
  SeedArena::mine().reset();
  std::printf("%zu %zu %zu\n", seeds, peak, held);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cuda = next((d for d in (os.environ.get("CUDA_HOME"), "/usr/local/cuda") if d and os.path.isdir(d)), None)
    if not shutil.which("g++") or not cuda:
        pytest.skip("no C++ compiler or CUDA headers")
    d = tmp_path_factory.mktemp("arena")
    (d / "arena.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "dcns_gb300", "csrc"), "-I",
                    os.path.join(cuda, "include"), str(d / "arena.cpp"), "-o", str(d / "arena")], check=True)
    return str(d / "arena")


@pytest.mark.parametrize("depth,windows", [(1, 1), (40, 100), (1500, 3), (3000, 1)])
def test_blocks_hold_the_nodes_alive(program, depth, windows):
    out = subprocess.run([program, str(depth), str(windows)], capture_output=True, text=True, check=True).stdout
    seeds, peak, held = (int(v) for v in out.split())
    assert seeds == depth * (windows + 1)
    # alive at once: the sets of two neighbouring levels and those above (one seed each), the window's, the pair's:
    # under 5 sets of `depth` nodes of 48 bytes; blocks double, so under four times that; the first block is 256 KB
    assert peak <= (256 << 10) + 4 * 5 * 48 * depth + 4096, peak
    assert held <= (256 << 10) + 4096, held
