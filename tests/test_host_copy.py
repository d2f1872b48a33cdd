"""The copies of pageable images through a ring of pinned memory (csrc/host_copy.h), on the CPU: the copy engine is a fake whose
copies are done at once or some time later, the helper threads may not be had, and a copy may be refused."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nncv_b200", "csrc")
CUDA = os.path.dirname(os.path.dirname(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"))

PROGRAM = r"""
#include <cuda_runtime.h>
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <vector>

// ---- the fake: a copy is carried out when its event has been asked for `late` times
static int late = 0, refuse_at = -1, copies = 0, threads_left = 1000;
struct Pending { void* d; const void* s; size_t n; };
static std::vector<Pending> unrecorded;
static std::map<void*, std::pair<int, std::vector<Pending>>> events;
static void carry_out(std::vector<Pending>& v) {
  for (auto& p : v) memcpy(p.d, p.s, p.n);
  v.clear();
}
extern "C" {
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned int) { return (*p = malloc(n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned int) { *e = (cudaEvent_t)malloc(1); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { carry_out(events[e].second); events.erase(e); free(e); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  if (copies++ == refuse_at) return cudaErrorInvalidValue;
  unrecorded.push_back({d, s, n});
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
  auto& v = events[e];
  v.first = late;
  for (auto& p : unrecorded) v.second.push_back(p);
  unrecorded.clear();
  return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) {
  auto& v = events[e];
  if (!v.second.empty() && v.first-- > 0) return cudaErrorNotReady;
  carry_out(v.second);
  return cudaSuccess;
}
int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* x) {
  if (threads_left-- <= 0) return EAGAIN;
  static auto real = (int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*))dlsym(RTLD_NEXT, "pthread_create");
  return real(t, a, f, x);
}
}
#include "host_copy.h"

int main(int argc, char** argv) {
  threads_left = atoi(argv[1]);
  late = atoi(argv[2]);
  const int refuse = atoi(argv[3]);
  nncv_b200::HostCopier c;
  unsigned seed = 1;
  for (size_t bytes : {(size_t)1, (size_t)524288, (size_t)524289, (size_t)(20 << 20) + 12345, (size_t)(3 << 20)}) {
    std::vector<unsigned char> src(bytes), dst(bytes);
    for (auto& b : src) b = (unsigned char)((seed = seed * 1664525u + 1013904223u) >> 24);
    for (int again = 0; again < 3; ++again) {
      std::fill(dst.begin(), dst.end(), 0);
      copies = 0;
      const long pieces = (long)((bytes + 524287) / 524288);
      refuse_at = again == 1 && refuse < pieces ? refuse : -1;
      const cudaError_t e = c.copy(dst.data(), src.data(), bytes, nullptr);
      if (e != (refuse_at >= 0 ? cudaErrorInvalidValue : cudaSuccess)) return printf("status %d of %zu bytes\n", (int)e, bytes), 1;
      for (auto& v : events) carry_out(v.second.second);   // the stream is waited for
      unrecorded.clear();
      if (e == cudaSuccess && dst != src) return printf("%zu bytes, pass %d: wrong\n", bytes, again), 1;
    }
  }
  puts("ok");
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if not shutil.which("g++") or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("host_copy")
    (d / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-rdynamic", "-I", CSRC, "-I", os.path.join(CUDA, "include"), str(d / "t.cpp"), "-o", str(d / "t"),
                    "-lpthread", "-ldl"], check=True, timeout=300)
    return str(d / "t")


@pytest.mark.parametrize("threads", [1000, 1, 0])
@pytest.mark.parametrize("late", [0, 40])
@pytest.mark.parametrize("refuse", [1000, 0, 5])
def test_every_byte_arrives_or_the_error_is_said(program, threads, late, refuse):
    r = subprocess.run([program, str(threads), str(late), str(refuse)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stdout, r.stderr[-500:])
