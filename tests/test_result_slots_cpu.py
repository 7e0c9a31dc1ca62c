"""The result slots of blocking probes (csrc/result_slot.hpp) against fake CUDA
calls: bounded, given back, remade after a failure, and with no call that
allocates or frees outside the relaxed capture mode (in the default one it
would end a stream capture that another thread has open)."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bloomfilter-bsd_b200", "csrc")

FAKE = r"""
#pragma once
#include <cstddef>
#include <cstdlib>
enum cudaError_t { cudaSuccess, cudaErrorMemoryAllocation };
enum cudaStreamCaptureMode { cudaStreamCaptureModeGlobal, cudaStreamCaptureModeThreadLocal, cudaStreamCaptureModeRelaxed };
constexpr unsigned cudaHostAllocMapped = 1, cudaHostAllocPortable = 2;
inline thread_local cudaStreamCaptureMode mode = cudaStreamCaptureModeGlobal;
inline int unsafe_calls = 0, live = 0, fail_at = -1;
inline cudaError_t fake_call() {
  if (mode != cudaStreamCaptureModeRelaxed) unsafe_calls++;
  return fail_at-- == 0 ? cudaErrorMemoryAllocation : cudaSuccess;
}
inline cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode* m) {
  const cudaStreamCaptureMode old = mode;
  mode = *m;
  *m = old;
  return cudaSuccess;
}
template <class T>
cudaError_t cudaMalloc(T** p, size_t n) {
  if (fake_call()) return cudaErrorMemoryAllocation;
  live++;
  *p = static_cast<T*>(std::malloc(n));
  return cudaSuccess;
}
inline cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMalloc(p, n); }
inline cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) { *d = h; return fake_call(); }
inline cudaError_t cudaFree(void* p) { fake_call(); live--; std::free(p); return cudaSuccess; }
inline cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
"""

MAIN = r"""
#include "result_slot.hpp"
#include <cstdio>
#include <set>
#include <utility>
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
using dtlg::ResultSlot;
using dtlg::ResultSlots;
static_assert(noexcept(std::declval<ResultSlots&>().acquire(1)), "");
static_assert(noexcept(std::declval<ResultSlots&>().release(nullptr)), "");
static_assert(noexcept(std::declval<ResultSlots&>().drop(nullptr)), "");
int main() {
  ResultSlots r;
  ResultSlot* s[ResultSlots::kMax];
  std::set<ResultSlot*> seen;
  for (auto& x : s) {
    x = r.acquire(256);
    CHECK(x && x->dev && x->host && x->host[0] == 0 && x->fresh);
    seen.insert(x);
  }
  CHECK(seen.size() == ResultSlots::kMax && r.acquire(256) == nullptr);
  s[3]->ticket = 7;
  r.release(s[3]);
  CHECK(r.acquire(256) == s[3] && s[3]->ticket == 7);  // kept as it was
  r.drop(s[5]);
  CHECK(live == 2 * ResultSlots::kMax - 2);
  for (int at = 0; at < 3; at++) {                     // each call of the making fails once
    fail_at = at;
    CHECK(r.acquire(256) == nullptr && live == 2 * ResultSlots::kMax - 2);
  }
  fail_at = -1;
  s[5] = r.acquire(256);
  CHECK(s[5] && s[5]->fresh && s[5]->ticket == 0 && r.acquire(256) == nullptr);
  for (auto& x : s) r.drop(x);
  CHECK(live == 0 && unsafe_calls == 0 && mode == cudaStreamCaptureModeGlobal);
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_slots_with_fake_cuda_calls(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(FAKE)
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "slots"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{tmp_path}", f"-I{CSRC}", str(tmp_path / "main.cpp"), "-o", str(exe),
                    "-lpthread"], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout
