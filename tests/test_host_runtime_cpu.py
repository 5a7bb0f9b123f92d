"""How a context meets the CUDA runtime on its error paths (common.cuh), against a fake runtime that
records its calls: no GPU."""
import ctypes
import os
import subprocess

import pytest

from conftest import PKG, ROOT

FAKE = r"""
#pragma once
#include <cstddef>
#include <vector>
typedef struct FakeStream* cudaStream_t;
typedef struct FakeEvent* cudaEvent_t;
enum cudaError_t { cudaSuccess = 0, cudaErrorMemoryAllocation = 2, cudaErrorNotReady = 600, cudaErrorUnknown = 999 };
constexpr unsigned cudaEventDisableTiming = 2;
extern std::vector<cudaStream_t> g_synced;
extern cudaError_t g_query, g_last;
extern unsigned* g_status;
inline cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  g_synced.push_back(s);
  if (g_status) *g_status |= 1;  // a kernel that was still running reports late
  return cudaSuccess;
}
inline cudaError_t cudaStreamQuery(cudaStream_t) { return g_last = g_query; }
inline cudaError_t cudaGetLastError() { const cudaError_t e = g_last; g_last = cudaSuccess; return e; }
inline const char* cudaGetErrorString(cudaError_t) { return "fake"; }
inline cudaError_t cudaMalloc(void**, size_t) { return cudaErrorMemoryAllocation; }
inline cudaError_t cudaFree(void*) { return cudaSuccess; }
inline cudaError_t cudaMallocHost(void**, size_t) { return cudaErrorMemoryAllocation; }
inline cudaError_t cudaFreeHost(void*) { return cudaSuccess; }
inline cudaError_t cudaEventCreate(cudaEvent_t*) { return cudaSuccess; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t*, unsigned) { return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
"""

SRC = r"""
#include "common.cuh"
#include <algorithm>
std::vector<cudaStream_t> g_synced;
cudaError_t g_query = cudaSuccess, g_last = cudaSuccess;
unsigned* g_status = nullptr;
namespace bg { std::atomic<uint64_t> g_launches{0}; }
using namespace bg;
static cudaStream_t st(size_t i) { return reinterpret_cast<cudaStream_t>(16 * (i + 1)); }
// a call that throws after its first launches, or does not: streams waited for, the error word after
// it, and whether the exception came through
extern "C" int t_drained(int fail, int* synced, unsigned* status) {
  Ctx c;
  unsigned word = 0;
  c.d_status = &word;
  g_status = &word;
  c.stream = st(0);
  c.copy = st(1);
  for (int i = 0; i < kStreams; i++) c.side[i] = st(2 + i);
  g_synced.clear();
  int seen = 0;
  try {
    drained(c, [&] { if (fail) c.ws.get("scratch", 1 << 20); });  // the allocation fails
  } catch (const Error& e) {
    seen = e.status;
  }
  g_status = nullptr;
  *status = word;
  *synced = 0;
  for (int i = 0; i < 2 + kStreams; i++) *synced += std::count(g_synced.begin(), g_synced.end(), st(i)) > 0;
  return seen;
}
// what stream_drained says of a query's result (2: it throws), and the last error it leaves
extern "C" int t_stream_drained(int query, int* last) {
  g_query = (cudaError_t)query;
  int r = 2;
  try {
    r = stream_drained(st(0)) ? 1 : 0;
  } catch (const Error&) {
  }
  *last = cudaGetLastError();
  return r;
}
"""


def build(tmp_path, src):
    fake = tmp_path / "fake"
    fake.mkdir()
    (fake / "cuda_runtime.h").write_text(FAKE)
    (tmp_path / "t.cpp").write_text(src)
    so = str(tmp_path / "t.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", str(fake), "-I", os.path.join(PKG, "csrc"),
                    "-I", os.path.join(ROOT, "include"), "-x", "c++", "-o", so, str(tmp_path / "t.cpp")], check=True)
    return ctypes.CDLL(so)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return build(tmp_path_factory.mktemp("host_runtime"), SRC)


def test_a_failed_call_leaves_nothing_in_flight(lib):
    """every stream of the context is waited for before the error reaches the caller, and an error
    flag that a kernel raises meanwhile does not fail the next call; a call that succeeds waits for
    nothing here"""
    synced, status = ctypes.c_int(), ctypes.c_uint()
    E_OOM, streams = 2, 9
    assert lib.t_drained(1, ctypes.byref(synced), ctypes.byref(status)) == E_OOM
    assert (synced.value, status.value) == (streams, 0)
    assert lib.t_drained(0, ctypes.byref(synced), ctypes.byref(status)) == 0
    assert synced.value == 0


def test_a_stream_still_running_is_no_error(lib):
    last = ctypes.c_int()
    assert (lib.t_stream_drained(600, ctypes.byref(last)), last.value) == (0, 0)
    assert (lib.t_stream_drained(0, ctypes.byref(last)), last.value) == (1, 0)
    assert lib.t_stream_drained(999, ctypes.byref(last)) == 2


def test_cached_numbers_are_shared_without_a_race(tmp_path):
    """what lanes compute at the same first use, under the thread sanitizer"""
    src = SRC + r"""
#include <thread>
int main() {
  static CachedInt cache[4];
  std::vector<std::thread> t;
  std::atomic<int> bad{0};
  for (int i = 0; i < 8; i++)
    t.emplace_back([&] {
      for (int k = 0; k < 4000; k++)
        if (cache[k % 4].get([&] { return 7 + k % 4; }) != 7 + k % 4) bad++;
    });
  for (auto& x : t) x.join();
  return bad.load();
}
"""
    fake = tmp_path / "fake"
    fake.mkdir()
    (fake / "cuda_runtime.h").write_text(FAKE)
    (tmp_path / "t.cpp").write_text(src)
    exe = str(tmp_path / "t")
    made = subprocess.run(["g++", "-O1", "-g", "-std=c++17", "-fsanitize=thread", "-pthread", "-I", str(fake), "-I",
                           os.path.join(PKG, "csrc"), "-x", "c++", "-o", exe, str(tmp_path / "t.cpp")],
                          capture_output=True, text=True)
    if made.returncode and "tsan" in made.stderr:
        pytest.skip("no thread sanitizer here")
    assert made.returncode == 0, made.stderr[-2000:]
    out = subprocess.run([exe], capture_output=True, text=True)
    if "unexpected memory mapping" in out.stderr:  # the sanitizer and this kernel's address randomisation
        out = subprocess.run(["setarch", "-R", exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stderr[-2000:]
