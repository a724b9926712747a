"""The pool of pinned chunks behind pageable copies, on the host with a fake CUDA
runtime that counts: objects that copy again and again on several threads' behalf
page-lock once each and not in every round of calls, a second device's pairs have
their own place, chunks are released outside the pool's lock, and what is kept
when the users are gone is two pairs a device."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cstdio>
#include <cstdlib>
#include <memory>
#include <thread>
#include <vector>
#include "host_staging.h"
using namespace cgx_staging;

static int g_device = 0, g_locked = 0, g_live = 0, g_free_under_lock = 0;
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = g_device; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t) { ++g_locked; ++g_live; *p = std::malloc(16); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) {
  std::thread([] { if (chunk_pool().mu.try_lock()) chunk_pool().mu.unlock(); else ++g_free_under_lock; }).join();
  --g_live; std::free(p); return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)std::malloc(1); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { a->type = cudaMemoryTypeHost; return cudaSuccess; }
}

#ifdef HAVE_USERS
using Owner = User;
#else
struct Owner { explicit Owner(int) {} };
#endif

// `n` objects on `device` that each take a pair, hold it together and give it back
static void round_of_calls(int device, int n) {
  g_device = device;
  std::vector<std::unique_ptr<Staging>> all;
  for (int i = 0; i < n; ++i) {
    all.emplace_back(new Staging(nullptr));
    if (all.back()->init() != cudaSuccess) std::exit(2);
  }
}

int main() {
  {
    std::vector<std::unique_ptr<Owner>> owners;
    for (int d = 0; d < 2; ++d)
      for (int i = 0; i < 5; ++i) owners.emplace_back(new Owner(d));
    for (int d = 0; d < 2; ++d) round_of_calls(d, 5);
    const int first = g_locked;
    for (int k = 0; k < 20; ++k) round_of_calls(k & 1, 5);
    std::printf("first %d later %d kept %d", first, g_locked - first, g_live);
  }
  const int gone = g_live;
  g_locked = 0;
  for (int k = 0; k < 4; ++k) round_of_calls(k & 1, 1);
  std::printf(" after %d transient %d underlock %d\n", gone, g_locked, g_free_under_lock);
}
"""


def cuda_include():
    for d in ("/usr/local/cuda/include", os.path.join(os.path.dirname(os.path.dirname(shutil.which("nvcc") or "/x/x")), "include")):
        if os.path.exists(os.path.join(d, "cuda_runtime.h")):
            return d
    pytest.skip("no CUDA headers")


def test_pairs_are_locked_once(tmp_path):
    src = tmp_path / "pool.cpp"
    src.write_text(SRC)
    exe = str(tmp_path / "pool")
    subprocess.run(["/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++", "-std=c++17", "-O1", "-DHAVE_USERS",
                    "-I", os.path.join(ROOT, "nextgen_b200", "csrc"), "-I", cuda_include(), str(src), "-o", exe, "-lpthread"],
                   check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout
    assert out.split() == "first 20 later 0 kept 20 after 8 transient 0 underlock 0".split(), out
