"""The seed-scan filter's tile count, on the host: the arithmetic that the device's plan and scan share (common.h), with
the numbers of sequences that are marked everywhere.  Two repeats of 3 Mb want 187,500 window pairs x 11,719 tiles, more
than 2^31: the list stays incomplete in the reader's eyes, and no tile is written outside it."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include <cstdint>
#include <cstdio>
#include <type_traits>
#include "common.h"
int main() {
  using Count = std::remove_reference_t<decltype(*dcns::FiltTiles::count)>;
  const int32_t cap = 1 << 20;
  const struct { int64_t duos; int32_t tiles; } cases[] = {{4, 250}, {1024, 1024}, {1024, 1025}, {187500, 11719},
                                                            {1 << 20, 699051}};
  for (const auto &c : cases) {
    Count wanted = 0;
    int64_t written = 0, outside = 0;
    for (int64_t d = 0; d < c.duos; ++d) {
      const Count at = wanted;
      wanted += (Count)c.tiles;
      for (const int32_t k : {0, c.tiles - 1}) {  // first and last of the duo's tiles
        const int32_t p = dcns::filt_place(at, k, cap);
        if (p >= 0) ++written;
        if (p >= cap || (p >= 0 && (uint64_t)p != (uint64_t)(d * c.tiles + k))) ++outside;
      }
    }
    std::printf("%lld %d %lld %lld\n", (long long)(c.duos * c.tiles), (int)dcns::filt_listed(wanted, cap),
                (long long)written, (long long)outside);
  }
}
"""


def test_tile_counts_beyond_an_int(tmp_path):
    cuda = next((d for d in (os.environ.get("CUDA_HOME"), "/usr/local/cuda") if d and os.path.isdir(d)), None)
    if not shutil.which("g++") or not cuda:
        pytest.skip("no C++ compiler or CUDA headers")
    src, exe = tmp_path / "count.cpp", tmp_path / "count"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "dcns_gb300", "csrc"), "-I",
                    os.path.join(cuda, "include"), str(src), "-o", str(exe)], check=True)
    rows = [[int(v) for v in line.split()]
            for line in subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.splitlines()]
    assert len(rows) == 5
    for total, listed, written, outside in rows:
        assert listed == (total <= 1 << 20) and outside == 0 and written > 0, total
