"""HostCopier (csrc/host_copy.h) on the CPU, over a stand-in for the CUDA
runtime whose copies are memcpy: contents of random scattered pieces both ways,
a call that does not wait for helper threads which wake late, and copies where
no pinned memory, no event or no thread can be had."""
import shutil
import subprocess
from pathlib import Path

import pytest

from signed_triangle_counting_b200 import build

CUDA = r"""
#pragma once
#include <cstdlib>
#include <cstring>
typedef int cudaError_t;
typedef void* cudaStream_t;
typedef int* cudaEvent_t;
enum { cudaSuccess = 0, cudaErrorMemoryAllocation = 2 };
enum { cudaMemcpyHostToDevice, cudaMemcpyDeviceToHost };
enum { cudaEventDisableTiming };
enum { cudaMemoryTypeUnregistered, cudaMemoryTypeHost };
struct cudaPointerAttributes { int type; };
inline int cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { a->type = 0; return 0; }
inline int cudaGetLastError() { return 0; }
inline bool fail_pinned = false;
inline int fail_events = -1;  // events that can still be made (-1: all)
inline int cudaMallocHost(void** p, size_t n) {
  if (fail_pinned) return cudaErrorMemoryAllocation;
  *p = malloc(n);
  return 0;
}
inline int cudaFreeHost(void* p) { free(p); return 0; }
inline int cudaEventCreateWithFlags(cudaEvent_t* e, int) {
  if (fail_events == 0) return cudaErrorMemoryAllocation;
  if (fail_events > 0) fail_events--;
  *e = new int(0);
  return 0;
}
inline int cudaEventSynchronize(cudaEvent_t e) { return e ? 0 : 400; }
inline int cudaEventDestroy(cudaEvent_t e) { delete e; return 0; }
inline int cudaEventRecord(cudaEvent_t, cudaStream_t) { return 0; }
inline int cudaStreamSynchronize(cudaStream_t) { return 0; }
inline int cudaMemcpyAsync(void* d, const void* s, size_t n, int, cudaStream_t) { memcpy(d, s, n); return 0; }
"""

PROGRAM = r"""
#include <dlfcn.h>
#include <pthread.h>
#include <unistd.h>

#include <cstdio>
#include <random>
#include <string>

#include "host_copy.h"

static bool late = false;
static pthread_t main_thread;
// Helper threads come back from a wait 400 ms after they were woken.
extern "C" int pthread_cond_wait(pthread_cond_t* c, pthread_mutex_t* m) {
  using F = int (*)(pthread_cond_t*, pthread_mutex_t*);
  static F real = (F)dlsym(RTLD_NEXT, "pthread_cond_wait");
  const int r = real(c, m);
  if (late && !pthread_equal(pthread_self(), main_thread)) {
    pthread_mutex_unlock(m);
    usleep(400000);
    pthread_mutex_lock(m);
  }
  return r;
}
static bool fail_threads = false;
extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* x) {
  using F = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
  static F real = (F)dlsym(RTLD_NEXT, "pthread_create");
  return fail_threads ? EAGAIN : real(t, a, f, x);
}
namespace stc {
void cuda_check(cudaError_t e, const char* what) { if (e) throw std::string(what); }
}

static std::mt19937_64 rng(1);
static bool round_trip(stc::HostCopier& c, const std::vector<size_t>& sizes, bool reverse) {
  std::vector<std::vector<char>> h;
  size_t total = 0, at = 0;
  for (size_t n : sizes) {
    h.emplace_back(n);
    for (size_t i = 0; i < n; i += 97) h.back()[i] = (char)rng();
    total += n;
  }
  std::vector<char> dev(total + 1);
  std::vector<stc::HostCopier::Piece> p;
  for (auto& x : h) p.push_back({dev.data() + at, x.data(), x.size()}), at += x.size();
  if (reverse) std::reverse(p.begin(), p.end());
  c.upload(p, nullptr);
  at = 0;
  for (auto& x : h) {
    if (x.size() && memcmp(dev.data() + at, x.data(), x.size())) return false;
    at += x.size();
  }
  const auto want = h;
  for (auto& x : h) std::fill(x.begin(), x.end(), 0);
  c.download(p, nullptr);
  return h == want;
}

int main(int argc, char** argv) {
  main_thread = pthread_self();
  const std::string mode = argv[1];
  stc::HostCopier c;
  if (mode == "random") {
    for (int it = 0; it < 60; it++) {
      std::vector<size_t> sizes(1 + rng() % 40);
      for (auto& n : sizes) n = rng() % (it % 3 ? 300000 : 30000000 / sizes.size());
      if (!round_trip(c, sizes, it & 1)) return printf("contents differ (%d)\n", it), 1;
      if (it % 25 == 7) c.release();
    }
  } else if (mode == "late") {
    if (!round_trip(c, {24u << 20}, false)) return 1;  // makes the threads
    usleep(200000);                                    // all of them wait
    late = true;
    for (size_t n : {3u << 20, 24u << 20}) {
      std::vector<char> dev(n), host(n, 5);
      const auto t = std::chrono::steady_clock::now();
      c.upload({{dev.data(), host.data(), n}}, nullptr);
      c.download({{dev.data(), host.data(), n}}, nullptr);
      const double ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t).count();
      if (ms > 300) return printf("%zu bytes there and back took %.0f ms\n", n, ms), 1;
      usleep(600000);
    }
    late = false;
  } else if (mode == "scarce") {
    for (int what = 0; what < 3; what++) {
      fail_pinned = what == 0;
      fail_events = what == 1 ? 3 : -1;
      fail_threads = what == 2;
      for (int again = 0; again < 2; again++)
        if (!round_trip(c, {24u << 20, 5000, 3u << 20}, false)) return printf("contents differ (%d)\n", what), 1;
      fail_pinned = fail_threads = false;  // and once there is enough again
      fail_events = -1;
      if (!round_trip(c, {24u << 20, 5000, 3u << 20}, false)) return printf("contents differ (%d)\n", what), 1;
      c.release();
    }
  }
  puts("ok");
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory) -> Path:
    if shutil.which(build.HOST_CXX) is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("host_copy")
    (d / "cuda_runtime.h").write_text(CUDA)
    (d / "main.cpp").write_text(PROGRAM)
    subprocess.run([build.HOST_CXX, "-std=c++17", "-O2", "-Wall", f"-I{d}", f"-I{build.CSRC}",
                    str(d / "main.cpp"), "-o", str(d / "main"), "-pthread", "-ldl"], check=True)
    return d / "main"


@pytest.mark.parametrize("mode", ["random", "late", "scarce"])
def test_host_copier(program, mode):
    r = subprocess.run([str(program), mode], capture_output=True, text=True, timeout=120)
    assert (r.returncode, r.stdout) == (0, "ok\n"), r.stdout + r.stderr
