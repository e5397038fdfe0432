"""The cache of device blocks (csrc/gbfe_devcache.h) on a pretended device of 1,000 bytes: memory that a call has parked
itself is given back when an allocation of that call would fail, the cap holds, and threads may share a cache."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "dft-efe_gb300" / "csrc"
CUDA = Path(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc").resolve().parent.parent / "include"

SOURCE = r"""
#include "gbfe_devcache.h"
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <thread>
using namespace gbfe;
static std::mutex dev_mu;
static std::map<void *, size_t> dev;  // what is allocated
static size_t used = 0, frees = 0;
extern "C" cudaError_t cudaMalloc(void **p, size_t n) {
  std::lock_guard<std::mutex> lk(dev_mu);
  if (used + n > 1000) return cudaErrorMemoryAllocation;
  *p = malloc(1);
  dev[*p] = n;
  used += n;
  return cudaSuccess;
}
extern "C" cudaError_t cudaFree(void *p) {
  std::lock_guard<std::mutex> lk(dev_mu);
  if (!dev.count(p)) { printf("freed twice\n"); exit(1); }
  used -= dev[p];
  dev.erase(p);
  free(p);
  ++frees;
  return cudaSuccess;
}
extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }
#define CHECK(c) do { if (!(c)) { printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
int main() {
  void *a = nullptr, *b = nullptr, *c = nullptr;
  {
    DevCache cache;
    DevScope s{cache, 900};
    thread_dev_scope() = &s;
    // parked in this call, not yet synchronised: given back when the call needs the memory
    CHECK(dev_alloc(&a, 600) == cudaSuccess);
    dev_free(a, 600);
    CHECK(used == 600 && s.parked.size() == 1);
    CHECK(dev_alloc(&b, 700) == cudaSuccess);
    CHECK(used == 700 && s.parked.empty());
    // reused by exact size once safe
    dev_free(b, 700);
    s.mark_safe();
    CHECK(cache.bytes() == 700 && used == 700);
    CHECK(dev_alloc(&c, 700) == cudaSuccess && c == b && cache.bytes() == 0);
    // the cap counts what is parked and what the cache holds
    dev_free(c, 700);
    CHECK(dev_alloc(&a, 250) == cudaSuccess);
    dev_free(a, 250);
    CHECK(s.refused && used == 700);
    s.mark_safe();
    // another cache's blocks are given back too, and an impossible request still fails
    {
      DevCache other;
      DevScope t{other, 900};
      thread_dev_scope() = &t;
      CHECK(dev_alloc(&a, 800) == cudaSuccess && cache.bytes() == 0 && used == 800);
      CHECK(dev_alloc(&b, 300) == cudaErrorMemoryAllocation);
      dev_free(a, 800);
      t.mark_safe();
      thread_dev_scope() = nullptr;
      other.release();
      CHECK(used == 0 && other.bytes() == 0);
    }
    // threads on one cache
    std::atomic<int> bad{0};
    std::vector<std::thread> ts;
    for (int k = 0; k < 8; ++k)
      ts.emplace_back([&, k] {
        DevScope m{cache, 60};
        thread_dev_scope() = &m;
        for (int r = 0; r < 2000; ++r) {
          void *p = nullptr, *q = nullptr;
          if (dev_alloc(&p, 1 + (r + k) % 5) != cudaSuccess || dev_alloc(&q, 3) != cudaSuccess || p == q) ++bad;
          dev_free(p, 1 + (r + k) % 5);
          dev_free(q, 3);
          if (r % 7 == 0) m.mark_safe();
          if (r % 501 == 0) cache.release();
        }
        m.free_parked();
        thread_dev_scope() = nullptr;
      });
    for (auto &t : ts) t.join();
    CHECK(bad == 0 && cache.bytes() <= 60 && used == cache.bytes());
  }
  CHECK(used == 0 && dev.empty());
  return 0;
}
"""


def test_cache_of_device_blocks(tmp_path):
    if not shutil.which("g++") or not (CUDA / "cuda_runtime_api.h").exists():
        pytest.skip("g++ or the CUDA headers are not available")
    (tmp_path / "t.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=thread", "-pthread", f"-I{CSRC}", f"-I{CUDA}",
                    str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    r = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
