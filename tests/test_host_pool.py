"""The pool of page-locked blocks (csrc/host_pool.h), compiled against stand-ins for the CUDA calls it makes.
CPU only."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CUDA = Path(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc").resolve().parent.parent / "include"

PROGRAM = r"""
#include "host_pool.h"
#include <cstdio>
#include <cstdlib>
static int pinned = 0;
extern "C" cudaError_t cudaMallocHost(void** p, size_t n) { ++pinned; *p = std::malloc(n < 4096 ? n : 4096); return cudaSuccess; }
extern "C" cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
extern "C" cudaError_t cudaSetDevice(int) { return cudaSuccess; }
extern "C" cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
int main() {
  crb::PinnedPool pool;
  cudaError_t e;
  void* staging = pool.get(32u << 20, &e);
  pool.put(staging);
  for (int stream = 0; stream < 3; ++stream) {  // two small blocks beside the staging, three times
    void* a = pool.get(64, &e);
    void* b = pool.get(80, &e);
    void* s = pool.get(32u << 20, &e);
    if (s != staging || a == staging || b == staging) return 1;
    pool.put(s);
    pool.put(a);
    pool.put(b);
  }
  void* c = pool.get(200u << 10, &e);  // larger requests take any block up to 64 MiB over theirs
  if (c != staging) return 2;
  std::printf("%d", pinned);
  return 0;
}
"""


@pytest.mark.skipif(not (CUDA / "cuda_runtime.h").exists(), reason="no CUDA headers")
def test_small_requests_leave_large_blocks(tmp_path):
    src, exe = tmp_path / "pool.cpp", tmp_path / "pool"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", str(CUDA), "-I", str(ROOT / "cuda_replace_b200" / "csrc"),
                    "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert (r.returncode, r.stdout) == (0, "3")  # the staging block and two small ones
