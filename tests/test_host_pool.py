"""The host worker pool (engine.cpp HostPool): an item that throws in a worker thread is the caller's exception, as it is
in a loop on the caller's own thread, so that the C entry points return an error code for it."""
import os
import shutil
import subprocess

import pytest

import dcns_gb300

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <new>
#include <stdexcept>
#include "engine.h"
int main() {
  for (int64_t n : {2, 64, 5000}) {
    for (int64_t bad : {int64_t(-1), int64_t(0), n / 2, n - 1}) {
      std::atomic<int64_t> ran(0);
      const char *got = "none";
      try {
        dcns::host_parallel(n, [&](int64_t i) {
          ++ran;
          if (i == bad) throw std::bad_alloc();
        });
      } catch (const std::bad_alloc &) {
        got = "bad_alloc";
      }
      const bool ok = bad < 0 ? ran == n && got[0] == 'n' : ran <= n && got[0] == 'b';
      if (!ok) return std::printf("n %lld bad %lld: %s after %lld\n", (long long)n, (long long)bad, got, (long long)ran), 1;
    }
  }
  std::puts("ok");
}
"""


def test_an_item_that_throws_is_the_callers_exception(tmp_path):
    cuda = next((d for d in (os.environ.get("CUDA_HOME"), "/usr/local/cuda") if d and os.path.isdir(d)), None)
    if not shutil.which("g++") or not cuda:
        pytest.skip("no C++ compiler or CUDA headers")
    so = dcns_gb300.build()
    src, exe = tmp_path / "pool.cpp", tmp_path / "pool"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "dcns_gb300", "csrc"), "-I",
                    os.path.join(cuda, "include"), str(src), so, f"-Wl,-rpath,{os.path.dirname(so)}", "-lpthread", "-o",
                    str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stdout, r.stderr)
