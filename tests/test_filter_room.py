"""The seed-scan filter takes device memory that a call can do without: where the device has none left (another context
or library holds it), the call scans every window instead of failing.  The engine's host code runs here on a CUDA
runtime made of host memory, with a cap on what cudaMalloc gives and kernels that do nothing (no window is selected)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <unordered_map>
#include "engine.h"
static size_t cap = ~size_t(0), held = 0, most = 0;
static std::unordered_map<void *, size_t> blocks;
static int scans_all = 0, scans_marked = 0;
extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) {
  if (held + n > cap) return cudaErrorMemoryAllocation;
  *p = std::calloc(n, 1);
  blocks[*p] = n, held += n, most = std::max(most, held);
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) { return held -= blocks[p], blocks.erase(p), std::free(p), cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t n) { return *p = std::malloc(n), cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { return std::free(p), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  return std::memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { return std::memset(d, v, n), cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { return *f = *t = size_t(1) << 40, cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int) {
  return std::memset(p, 0, sizeof *p), p->major = 10, p->minor = 3, p->multiProcessorCount = 152, cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "an error"; }
cudaError_t cudaDeviceGetStreamPriorityRange(int *a, int *b) { return *a = *b = 0, cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int) { return *s = nullptr, cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 0, cudaSuccess; }
}
namespace dcns {
int scan_occupancy() { return 5; }
void launch_pack(const int8_t *, const int64_t *, const int64_t *, const int32_t *, int, uint32_t *, uint32_t *,
                 cudaStream_t) {}
void launch_filter(const FiltDesc &, Arena, Params, int, cudaStream_t) {}
void launch_filter_plan_l0(const FiltDesc &, L0Desc, int64_t, FiltTiles, int, cudaStream_t) {}
void launch_scan_tiles_l0(L0Desc, FiltTiles, Arena, Params, unsigned long long *, int *, int, cudaStream_t) {
  ++scans_marked;
}
void launch_scan_l0(L0Desc, int64_t, Arena, Params, unsigned long long *, int *, int64_t, cudaStream_t) { ++scans_all; }
void launch_l0_select(const unsigned long long *, int64_t, const int64_t *, const int2 *, int, const int64_t *, Arena,
                      Params, int *, int *, L0Rec *, int, cudaStream_t) {}
}  // namespace dcns
using namespace dcns;
// most memory that a call on a pair of n bases took (0: refused); limit: what cudaMalloc gives in all
static size_t call(int n, bool filter, size_t limit, int *marked) {
  cap = ~size_t(0), scans_all = scans_marked = 0;
  Context C;
  init_context(C, 0, 0);
  C.scan_filter = filter;
  cap = limit, most = held;
  dcns_params d{};
  d.match = 2, d.mismatch = -3, d.open1 = -4, d.ext1 = -2, d.open2 = -45, d.window = 38, d.min_score = 40, d.step = 8;
  d.w = 10, d.xdrop = 20, d.zdrop = 50, d.bandwidth = 20000, d.pvalue = .1, d.lambda = .38, d.kvalue = .007;
  std::vector<int8_t> a(n, 0), b(n, 1);
  std::vector<std::vector<FragOut>> out;
  try {
    for (int k = 0; k < 2; ++k) align_pairs(C, {PairIn{a.data(), n, b.data(), n}}, to_params(&d), 1, out);
  } catch (const Error &) {
    return 0;
  }
  *marked = scans_marked;
  return most;
}
int main() {
  for (int n : {3000, 40000, 150000}) {
    int m = 0;
    const size_t whole = call(n, false, ~size_t(0), &m), with = call(n, true, ~size_t(0), &m);
    if (!whole || with <= whole || m != 2) return std::printf("n %d: %zu %zu %d\n", n, whole, with, m), 1;
    // from what the call needs without the filter on, nothing is refused
    for (int k = 0; k <= 20; ++k) {
      const size_t limit = whole + (with - whole) * k / 20;
      if (!call(n, true, limit, &m)) return std::printf("n %d: refused with %zu of %zu\n", n, limit, with), 1;
      if (k == 20 && m != 2) return std::printf("n %d: the filter did not run\n", n), 1;
    }
  }
  std::puts("ok");
}
"""


def test_no_room_for_the_filter(tmp_path):
    cuda = next((d for d in (os.environ.get("CUDA_HOME"), "/usr/local/cuda") if d and os.path.isdir(d)), None)
    if not shutil.which("g++") or not cuda:
        pytest.skip("no C++ compiler or CUDA headers")
    csrc = os.path.join(ROOT, "dcns_gb300", "csrc")
    src, exe = tmp_path / "room.cpp", tmp_path / "room"
    src.write_text(PROGRAM)
    # the launchers of stages that no seed reaches stay unresolved
    subprocess.run(["g++", "-O1", "-std=c++17", "-w", "-I", csrc, "-I", os.path.join(cuda, "include"), str(src),
                    os.path.join(csrc, "engine.cpp"), "-no-pie", "-Wl,--unresolved-symbols=ignore-all", "-lpthread", "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stdout[-300:], r.stderr[-300:])
