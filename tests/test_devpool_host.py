"""The kept device memory (csrc/devpool.cu) on the host, over a stand-in for the runtime's
allocator: what is reused and by whom, the bound, what makes room, what is given back."""
import os
import subprocess

import pytest

from conftest import ROOT

CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include <set>
#include <vector>
#include "devpool.cu"
using namespace prbf;
static bool fail_new = false;
void* operator new(size_t n) {
  void* p = fail_new ? nullptr : std::malloc(n ? n : 1);
  if (!p) throw std::bad_alloc();
  return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }
static const size_t MB = (size_t)1 << 20, GB = (size_t)1 << 30;
static std::map<void*, size_t> live;   // what the driver has given out
static size_t taken = 0, capacity = 64 * GB;
static char* next_address = (char*)0x10000000;
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
  if (taken + n > capacity) return cudaErrorMemoryAllocation;
  *p = next_address;
  next_address += (n + 511) / 512 * 512;
  const bool f = fail_new;
  fail_new = false;  // (the stand-in's own bookkeeping)
  live[*p] = n;
  fail_new = f;
  taken += n;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  auto it = live.find(p);
  if (it == live.end()) { std::printf("freed twice or never allocated\n"); std::exit(2); }
  taken -= it->second;
  live.erase(it);
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return ""; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *f = capacity - taken; *t = capacity; return cudaSuccess; }
}
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
static void* get(size_t n) { void* p = nullptr; return dev_alloc(&p, n) == cudaSuccess ? p : nullptr; }
int main() {
  cudaStream_t s1 = (cudaStream_t)0x1, s2 = (cudaStream_t)0x2;
  {  // the same stream's block at once, another's only when that stream is done
    void *a, *b;
    { StreamScope sc(s1); a = get(3 * MB); dev_free(a); }
    { StreamScope sc(s2); b = get(3 * MB); CHECK(b != a); dev_free(b); }
    { StreamScope sc(s1); CHECK(get(3 * MB) == a); dev_free(a); }
    dev_pool_stream_done(0, s1);
    { StreamScope sc(s2); void* c = get(3 * MB); CHECK(c == b); void* d = get(3 * MB); CHECK(d == a);
      dev_free(c); dev_free(d); }
    CHECK(dev_pool_kept(0) == 6 * MB && taken == 6 * MB);
    CHECK(dev_mem_free() == capacity);  // kept blocks count as free
    dev_pool_trim(0);
    CHECK(dev_pool_kept(0) == 0 && taken == 0 && live.empty());
  }
  {  // outside of a context, and above the largest kept block: straight to the driver
    void* a = get(MB); dev_free(a); CHECK(taken == 0);
    StreamScope sc(s1);
    a = get(300 * MB); dev_free(a); CHECK(taken == 0 && dev_pool_kept(0) == 0);
  }
  {  // one context that changes sizes: the bound holds, and the newest sizes are the kept ones
    StreamScope sc(s1);
    for (int k = 0; k < 40; k++) {
      std::vector<void*> v;
      for (int j = 0; j < 4; j++) v.push_back(get((100 + 3 * k) * MB));
      for (void* p : v) dev_free(p);
      CHECK(dev_pool_kept(0) <= 2 * GB && dev_pool_kept(0) == taken);
    }
    CHECK(dev_pool_kept(0) > 2 * GB - 256 * MB);
    const size_t before = taken;
    std::vector<void*> v;
    for (int j = 0; j < 4; j++) v.push_back(get((100 + 3 * 39) * MB));
    CHECK(taken == before);  // all four from what is kept
    for (void* p : v) dev_free(p);
    for (int k = 0; k < 5; k++) { void* p = get(50 * MB); dev_free(p); }
    CHECK(dev_pool_kept(0) <= 2 * GB);
    void* p = get(50 * MB);
    const size_t t = taken;
    dev_free(p);
    CHECK(get(50 * MB) == p && taken == t);  // (a full pool still takes new blocks in)
    dev_free(p);
  }
  {  // a failed allocation empties what is kept and is tried again
    capacity = taken + 10 * MB;
    StreamScope sc(s2);
    void* p = get(200 * MB);
    CHECK(p != nullptr && dev_pool_kept(0) == 0);
    dev_free(p);
    void* big = get(GB);
    CHECK(big != nullptr);
    dev_free(big);
    CHECK(get(8 * GB) == nullptr);
    capacity = 64 * GB;
  }
  dev_pool_trim(0);
  CHECK(taken == 0);
  {  // sixteen contexts without a use
    { StreamScope sc(s1); void* a = get(MB); dev_free(a); }
    for (int k = 0; k < 16; k++) { dev_pool_stream_done(0, s2); CHECK(dev_pool_kept(0) == MB); }
    dev_pool_stream_done(0, s2);
    CHECK(dev_pool_kept(0) == 0 && taken == 0);
  }
  {  // blocks of a destroyed context are anyone's
    void* a;
    { StreamScope sc(s1, true); a = nullptr; }
    { StreamScope sc(s1); a = get(MB); }
    { StreamScope sc(s1, true); dev_free(a); }
    { StreamScope sc(s2); CHECK(get(MB) == a); dev_free(a); }
  }
  {  // no host memory: nothing is thrown at a destructor, nothing is lost
    StreamScope sc(s1);
    void *a = get(5 * MB), *b = get(6 * MB);
    dev_free(b);
    const size_t t = taken;
    fail_new = true;
    dev_free(a);  // (to the driver: it cannot be kept)
    dev_pool_stream_done(0, s2);
    fail_new = false;
    CHECK(taken == t - 5 * MB);
    fail_new = true;
    bool thrown = false;
    void *c = nullptr, *e = nullptr;
    try {
      dev_alloc(&c, 7 * MB);
    } catch (const std::bad_alloc&) {
      thrown = true;
    }
    CHECK(thrown && taken == t - 5 * MB && !c);
    try {
      thrown = false;
      dev_alloc(&e, 6 * MB);  // (a kept block: stays kept)
    } catch (const std::bad_alloc&) {
      thrown = true;
    }
    fail_new = false;
    CHECK(thrown && taken == t - 5 * MB && !e);
    CHECK(get(6 * MB) == b);
    dev_free(b);
  }
  CHECK(dev_pool_kept(7) == 0);
  dev_pool_trim(0);
  dev_pool_trim(7);
  CHECK(live.empty());
  std::printf("ok\n");
  return 0;
}
"""


def test_kept_memory(tmp_path):
    inc = os.path.join(CUDA, "include")
    if not os.path.exists(os.path.join(inc, "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    src, exe = str(tmp_path / "pool.cpp"), str(tmp_path / "pool")
    with open(src, "w") as f:
        f.write(SOURCE)
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-I", inc, "-I", os.path.join(ROOT, "petrbf_gb300", "csrc"), "-I",
                        os.path.join(ROOT, "include"), src, "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
