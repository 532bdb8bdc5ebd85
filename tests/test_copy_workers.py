"""The parallel host copy (csrc/host_pool.h): sizes around its parts, many threads at once. CPU only."""
import subprocess

import pytest

from tests.test_host_pool import CUDA, ROOT

PROGRAM = r"""
#include "host_pool.h"
#include <cstdio>
#include <cstdlib>
extern "C" cudaError_t cudaMallocHost(void** p, size_t n) { *p = std::malloc(n); return cudaSuccess; }
extern "C" cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
extern "C" cudaError_t cudaSetDevice(int) { return cudaSuccess; }
extern "C" cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
int main() {
  std::atomic<int> bad{0};
  auto work = [&](unsigned seed) {
    const size_t sizes[] = {0, 1, 4095, (1u << 20) - 1, 1u << 20, (1u << 20) + 1, (1u << 20) + 4097, 3u << 20, (9u << 20) + 12345};
    std::vector<unsigned char> src(10u << 20), dst(10u << 20);
    for (int round = 0; round < 40; ++round) {
      const size_t n = sizes[(seed + round) % 9];
      for (size_t i = 0; i < n + 64; ++i) src[i] = (unsigned char)(i * 2654435761u >> 13 ^ (seed + round));
      memset(dst.data(), 0x5A, n + 64);
      crb::parallel_memcpy(dst.data(), src.data(), n);
      if (memcmp(dst.data(), src.data(), n)) ++bad;
      for (size_t i = n; i < n + 64; ++i) bad += dst[i] != 0x5A;
    }
  };
  work(0);
  std::vector<std::thread> th;
  for (unsigned t = 0; t < 6; ++t) th.emplace_back(work, t);
  for (auto& t : th) t.join();
  std::printf("%d", bad.load());
  return 0;
}
"""


@pytest.mark.skipif(not (CUDA / "cuda_runtime.h").exists(), reason="no CUDA headers")
def test_copies_of_several_threads(tmp_path):
    src, exe = tmp_path / "copy.cpp", tmp_path / "copy"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", str(CUDA), "-I", str(ROOT / "cuda_replace_b200" / "csrc"),
                    "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert (r.returncode, r.stdout) == (0, "0")
