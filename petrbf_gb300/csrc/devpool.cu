// devpool.cu -- device memory kept between uses. A cudaMalloc and cudaFree pair costs 60 us
// (430 us at 512 MB), and a one-shot call (its own context, some thirty buffers) spent most of its
// time in them: evaluating 4.9x10^5 sources at 3x10^5 points took 3.6 ms, 1.4 of them kernels, and
// 1.7 with the pool; the 10^4-point solve in a context of its own 35.4 -> 34.3 ms.
//
// A freed block may still be read by work its stream has queued, so it carries that stream (the
// context's, set for the length of a call, StreamScope) and serves the same stream again at once,
// ordered behind that work; other streams get it once its own is known to be idle
// (dev_pool_stream_done, when the context is destroyed). Calls outside of any context allocate and
// free as before. Bounded: blocks up to kMaxBlock, kMaxCached bytes per device, beyond which the
// blocks that have lain longest make room. Given back when an allocation fails, when 16 contexts
// have come and gone without a use, and on request (prbf_memory_release). What is kept counts as
// free memory where a size is chosen by it (dev_mem_free), so that no choice depends on the calls
// that came before.
#include <map>
#include <mutex>
#include <new>
#include <unordered_map>
#include <vector>

#include "device.h"

namespace prbf {
namespace {

constexpr size_t kMaxBlock = (size_t)256 << 20, kMaxCached = (size_t)2 << 30;
constexpr unsigned long long kKeep = 16;

thread_local cudaStream_t t_stream = nullptr;
thread_local bool t_on = false, t_idle = false;

struct Free {
  void* p;
  cudaStream_t stream;       // may still have work on the block; null: idle
  unsigned long long since;  // contexts destroyed when it was freed
  unsigned long long turn;   // frees before it
};

struct DevicePool {
  std::multimap<size_t, Free> free;
  size_t cached = 0;
  unsigned long long epoch = 0;  // contexts destroyed
  unsigned long long turn = 0;   // blocks freed
};

struct Pool {
  std::mutex m;
  std::map<int, DevicePool> dev;
  std::unordered_map<void*, std::pair<int, size_t>> used;  // blocks of the pool in use: device, size
};

Pool& pool() {
  static Pool* p = new Pool();  // (outlives every static buffer's destructor)
  return *p;
}

size_t size_class(size_t b) {  // eight classes per power of two
  if (b <= 512) return 512;
  size_t step = 64;
  while (step * 16 <= b) step *= 2;
  return (b + step - 1) / step * step;
}

int current_device() {
  int d = 0;
  PRBF_CUDA(cudaGetDevice(&d));
  return d;
}

// Takes the device's cached blocks out (all, or those unused for long), for the caller to free.
std::vector<void*> take(DevicePool& D, bool all) {
  std::vector<void*> out;
  out.reserve(D.free.size());  // (whatever fails, fails before a block is taken out)
  for (auto it = D.free.begin(); it != D.free.end();)
    if (all || D.epoch - it->second.since > kKeep) {
      out.push_back(it->second.p);
      D.cached -= it->first;
      it = D.free.erase(it);
    } else {
      ++it;
    }
  return out;
}

// Takes out the blocks that have lain longest until a block of cls bytes fits beside the rest.
void make_room(DevicePool& D, size_t cls, std::vector<void*>& out) {
  while (D.cached + cls > kMaxCached) {
    auto old = D.free.begin();
    for (auto it = D.free.begin(); it != D.free.end(); ++it)
      if (it->second.turn < old->second.turn) old = it;
    out.push_back(old->second.p);
    D.cached -= old->first;
    D.free.erase(old);
  }
}

}  // namespace

StreamScope::StreamScope(cudaStream_t s, bool idle) : stream(t_stream), on(t_on), was_idle(t_idle) {
  t_stream = s;
  t_on = true;
  t_idle = idle;
}

StreamScope::~StreamScope() {
  t_stream = stream;
  t_on = on;
  t_idle = was_idle;
}

cudaError_t dev_alloc(void** p, size_t bytes) {
  const size_t cls = size_class(bytes);
  if (!t_on || cls > kMaxBlock) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();
    dev_pool_trim(current_device());
    return cudaMalloc(p, bytes);
  }
  Pool& P = pool();
  const int d = current_device();
  {
    std::lock_guard<std::mutex> lk(P.m);
    DevicePool& D = P.dev[d];
    auto r = D.free.equal_range(cls);
    auto best = r.second;
    for (auto it = r.first; it != r.second; ++it) {
      if (it->second.stream && it->second.stream != t_stream) continue;
      best = it;
      if (it->second.stream) break;  // the same stream's first
    }
    if (best != r.second) {
      P.used[best->second.p] = {d, cls};  // (may throw: *p is set last)
      *p = best->second.p;
      D.cached -= cls;
      D.free.erase(best);
      return cudaSuccess;
    }
  }
  cudaError_t e = cudaMalloc(p, cls);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    dev_pool_trim(d);
    return cudaMalloc(p, bytes);  // (as asked for; not the pool's)
  }
  if (e == cudaSuccess) {
    try {
      std::lock_guard<std::mutex> lk(P.m);
      P.used[*p] = {d, cls};
    } catch (const std::bad_alloc&) {
      cudaFree(*p);
      *p = nullptr;
      throw;
    }
  }
  return e;
}

void dev_free(void* p) {
  Pool& P = pool();
  std::vector<void*> out;  // (cudaFree waits for work on what it frees, whatever its stream)
  try {
    std::lock_guard<std::mutex> lk(P.m);
    auto it = P.used.find(p);
    if (it != P.used.end()) {
      const auto [d, cls] = it->second;
      P.used.erase(it);
      if (t_on) {
        DevicePool& D = P.dev[d];
        make_room(D, cls, out);
        D.free.insert({cls, Free{p, t_idle ? nullptr : t_stream, D.epoch, D.turn++}});
        D.cached += cls;
        p = nullptr;
      }
    }
  } catch (const std::bad_alloc&) {  // (buffers are freed by destructors)
  }
  if (p) cudaFree(p);
  for (void* q : out) cudaFree(q);
}

void dev_pool_stream_done(int device, cudaStream_t s) {
  Pool& P = pool();
  std::vector<void*> old;
  {
    std::lock_guard<std::mutex> lk(P.m);
    const auto it = P.dev.find(device);
    if (it == P.dev.end()) return;
    DevicePool& D = it->second;
    D.epoch++;
    for (auto& f : D.free)
      if (f.second.stream == s) f.second.stream = nullptr;
    try {
      old = take(D, false);
    } catch (const std::bad_alloc&) {  // (they go another time)
    }
  }
  for (void* p : old) cudaFree(p);
}

void dev_pool_trim(int device) {
  Pool& P = pool();
  std::vector<void*> all;
  {
    std::lock_guard<std::mutex> lk(P.m);
    const auto it = P.dev.find(device);
    if (it != P.dev.end()) all = take(it->second, true);
  }
  for (void* p : all) cudaFree(p);
}

size_t dev_pool_kept(int device) {
  Pool& P = pool();
  std::lock_guard<std::mutex> lk(P.m);
  const auto it = P.dev.find(device);
  return it == P.dev.end() ? 0 : it->second.cached;
}

size_t dev_mem_free() {
  size_t free_b = 0, total_b = 0;
  PRBF_CUDA(cudaMemGetInfo(&free_b, &total_b));
  return free_b + dev_pool_kept(current_device());
}

}  // namespace prbf
