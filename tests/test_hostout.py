"""Output staging (wavesim_b200/csrc/ws_hostout.h) on the CPU, over a stand-in for
the CUDA calls it makes: a stream is a list of copies that run when somebody
waits for it, so that what is still under way can be seen."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "wavesim_b200", "csrc")
CUDA_INC = "/usr/local/cuda/include"

FAKE = r"""
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>
#include <vector>
struct Copy { void* dst; const void* src; size_t n; };
static std::vector<Copy> queue;      // of the one stream
static std::recursive_mutex queue_mu;
static int host_allocs_left = 1 << 30, event_records_left = 1 << 30;
static int live = 0;                 // page-locked buffers
static std::atomic<int> news_left{1 << 30};
void* operator new(size_t n) {
  if (news_left-- <= 0) throw std::bad_alloc();
  return std::malloc(n);
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }
static void drain() {
  std::lock_guard<std::recursive_mutex> l(queue_mu);
  for (const Copy& c : queue) std::memcpy(c.dst, c.src, c.n);
  queue.clear();
}
static bool queued_into(const void* p, size_t n) {
  std::lock_guard<std::recursive_mutex> l(queue_mu);
  for (const Copy& c : queue)
    if ((char*)c.dst < (char*)p + n && (char*)p < (char*)c.dst + c.n) return true;
  return false;
}
extern "C" {
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  if (host_allocs_left-- <= 0) return cudaErrorMemoryAllocation;
  *p = std::malloc(n);
  ++live;
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { --live; std::free(p); return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::lock_guard<std::recursive_mutex> l(queue_mu);
  queue.push_back(Copy{d, s, n});
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { drain(); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)1; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) {
  return event_records_left-- <= 0 ? cudaErrorUnknown : cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { drain(); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
}
#include "ws_hostout.h"
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
"""

BODIES = {
    # an OutCopy given up between stage() and run(): the next taker of its buffer must not receive the copy
    "staged_and_given_up": r"""
  std::vector<char> src(1 << 20, 7), dst(1 << 20, 1);
  {
    ws::OutCopy c(dst.data(), dst.size(), 0);
    CHECK(c.ok());
    c.touch();
    CHECK(c.stage(src.data(), nullptr) == cudaSuccess);
  }
  size_t got = 0;
  void* p = ws::host_pool().get(dst.size(), &got);
  CHECK(p && !queued_into(p, got));
  ws::host_pool().put(p, got);
  CHECK(dst[5] == 1);
  return 0;""",
    # a chunk whose event could not be recorded is still under way
    "a_chunk_that_failed": r"""
  std::vector<char> src(9 << 20, 7), dst(9 << 20, 1);
  event_records_left = 0;
  {
    ws::OutCopy c(dst.data(), dst.size(), 0);
    c.touch();
    CHECK(c.stage(src.data(), nullptr) == cudaSuccess);
    CHECK(c.run() != cudaSuccess);
  }
  size_t got = 0;
  void* p = ws::host_pool().get(1, &got);
  CHECK(p && !queued_into(p, got));
  return 0;""",
    # groups of fields in a device buffer: the largest half, quarter, .. that fits, one field if need be, and no other error
    # taken for a lack of memory
    "groups_that_fit": r"""
  for (int room : {100, 16, 15, 5, 1}) {
    int tries = 0;
    cudaError_t e;
    const int g = ws::fitting_group(16, [&](int n) { ++tries; return n <= room ? cudaSuccess : cudaErrorMemoryAllocation; }, &e);
    CHECK(e == cudaSuccess && g <= room && g >= 1 && tries <= 5);
    CHECK(room < 16 || g == 16);
  }
  cudaError_t e;
  CHECK(ws::fitting_group(16, [](int) { return cudaErrorMemoryAllocation; }, &e) == 1 && e == cudaErrorMemoryAllocation);
  int tries = 0;
  ws::fitting_group(16, [&](int) { ++tries; return cudaErrorUnknown; }, &e);
  CHECK(e == cudaErrorUnknown && tries == 1);
  return 0;""",
    # no page-locked memory at all: through ordinary memory
    "no_page_locked_memory": r"""
  host_allocs_left = 0;
  for (size_t n : {(size_t)4097, (size_t)(9 << 20) + 13}) {
    std::vector<char> src(n, 7), dst(n, 1);
    ws::HostLease state(100);
    CHECK(state.p);
    ws::OutCopy c(dst.data(), n, 0);
    CHECK(c.ok());
    c.touch();
    CHECK(c.stage(src.data(), nullptr) == cudaSuccess);
    cudaStreamSynchronize(nullptr);
    CHECK(c.run() == cudaSuccess);
    CHECK(dst == src);
  }
  return 0;""",
    # no memory at any one of the allocations that staging a result makes: it arrives, or the call throws, but the
    # process goes on
    "no_memory": r"""
  std::vector<char> src(70 << 20, 7), dst(src.size(), 1);
  for (int k = 0; k < 40; ++k) {
    std::fill(dst.begin(), dst.end(), 1);
    news_left = k;
    bool arrived = false;
    try {
      ws::OutCopy c(dst.data(), dst.size(), 0);
      news_left = 1 << 30;
      c.touch();
      CHECK(c.stage(src.data(), nullptr) == cudaSuccess);
      arrived = c.run() == cudaSuccess;
    } catch (const std::bad_alloc&) {
    }
    news_left = 1 << 30;
    CHECK(!arrived || dst == src);
    // as the pool takes its buffers back
    void* p[3];
    size_t got[3];
    for (int i = 0; i < 3; ++i) p[i] = ws::host_pool().get(4096, &got[i]);
    news_left = k % 4;
    for (int i = 0; i < 3; ++i) ws::host_pool().put(p[i], got[i]);
    news_left = 1 << 30;
    ws::host_pool().trim();
    CHECK(live == 0);
  }
  return 0;""",
    # and the ordinary way, whole and in chunks
    "results_arrive": r"""
  for (size_t n : {(size_t)1, (size_t)4097, (size_t)(4 << 20), (size_t)(9 << 20) + 13, (size_t)(70 << 20)}) {
    std::vector<char> src(n, 7), dst(n, 1);
    ws::OutCopy c(dst.data(), n, 0);
    c.touch();
    CHECK(c.stage(src.data(), nullptr) == cudaSuccess);
    cudaStreamSynchronize(nullptr);
    CHECK(c.run() == cudaSuccess);
    CHECK(dst == src);
  }
  ws::host_pool().trim();
  CHECK(live == 0);
  return 0;""",
}


def run(tmp_path, body):
    src = tmp_path / "t.cpp"
    src.write_text(FAKE + "int main() {" + body + "\n}\n")
    exe = tmp_path / "t"
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", CSRC, "-I", CUDA_INC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA_INC), reason="needs g++ and CUDA headers")
@pytest.mark.parametrize("name", list(BODIES))
def test_buffers_and_results(tmp_path, name):
    run(tmp_path, BODIES[name])
