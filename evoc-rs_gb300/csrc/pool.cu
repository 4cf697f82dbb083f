// pool.cu — device buffers kept for reuse, one pool per context.
//
// The driver's stream-ordered allocator takes 1 to 2 us for a small buffer and
// about 1 us per megabyte for a large one that it has to map again (1.8 ms for the
// 1.9 GB of schedule planes at 2M points; 5 ms of a 32 ms pass in all, and half of a
// pass at 2,000 points). A call takes the same sizes as the one before, so freed
// buffers are kept by size class and handed out again. A pool belongs to one
// stream and only serves that stream, so a buffer's next use comes after its last
// one in stream order, as with the driver's allocator. A pool's free buffers are
// bounded by an eighth of the device's memory (the least recently freed go first), are
// given back when an allocation fails, and with the context. The bound is per context:
// contexts on one device hold as many eighths between them as there are contexts, and
// give them up to one another when an allocation fails.
//
// A pool is touched for another context only under the lock, only on the same device,
// and only while its stream is not being captured: a free enqueued then would become a
// part of the capture.
#include "evoc_internal.h"

#include <map>
#include <mutex>
#include <new>

namespace evoc {
namespace {

// Size classes: eight per octave from 512 bytes up.
size_t class_of(size_t bytes) {
  size_t step = 512;
  while (step * 16 < bytes) step *= 2;
  return (bytes + step - 1) / step * step;
}

struct Block {
  void* ptr;
  uint64_t stamp;  // order of freeing
};

struct Pool {
  std::map<size_t, std::vector<Block>> free_blocks;  // by size class
  size_t bytes = 0;                                  // free bytes held
  size_t limit = 0;
  uint64_t stamp = 0;
  int device = 0;
  bool capturing = false;  // the context is capturing its stream (dev_pool_capture)

  // A block of the class, or of a little more for buffers that are worth it.
  void* take(size_t cls, size_t* held) {
    const size_t most = cls >= ((size_t)1 << 20) ? cls + cls / 4 : cls;
    for (auto it = free_blocks.lower_bound(cls); it != free_blocks.end() && it->first <= most;
         ++it) {
      if (it->second.empty()) continue;
      void* p = it->second.back().ptr;
      it->second.pop_back();
      bytes -= it->first;
      *held = it->first;
      return p;
    }
    return nullptr;
  }
  // Gives buffers back until `to` bytes are left; one that cannot be freed stays.
  void shrink(size_t to, cudaStream_t s) {
    while (bytes > to) {
      auto oldest = free_blocks.end();
      for (auto it = free_blocks.begin(); it != free_blocks.end(); ++it)
        if (!it->second.empty() &&
            (oldest == free_blocks.end() ||
             it->second.front().stamp < oldest->second.front().stamp))
          oldest = it;
      if (oldest == free_blocks.end()) break;
      if (cudaFreeAsync(oldest->second.front().ptr, s) != cudaSuccess) {
        (void)cudaGetLastError();
        break;
      }
      oldest->second.erase(oldest->second.begin());
      bytes -= oldest->first;
    }
  }
};

std::mutex g_mu;
std::map<cudaStream_t, Pool> g_pools;

}  // namespace

void dev_pool_open(cudaStream_t s, int device, size_t limit) {
  std::lock_guard<std::mutex> lk(g_mu);
  Pool& p = g_pools[s];
  p.limit = limit;
  p.device = device;
}

void dev_pool_capture(cudaStream_t s, bool on) {
  std::lock_guard<std::mutex> lk(g_mu);
  auto it = g_pools.find(s);
  if (it != g_pools.end()) it->second.capturing = on;
}

void dev_pool_close(cudaStream_t s) {
  std::lock_guard<std::mutex> lk(g_mu);
  auto it = g_pools.find(s);
  if (it == g_pools.end()) return;
  it->second.shrink(0, s);
  g_pools.erase(it);
}

size_t dev_pool_bytes(cudaStream_t s) {
  std::lock_guard<std::mutex> lk(g_mu);
  auto it = g_pools.find(s);
  return it == g_pools.end() ? 0 : it->second.bytes;
}

// Bytes that dev_alloc could obtain for the stream: the device's free memory, what the
// driver's pool keeps of freed buffers (it returns none to the device), and what the
// contexts' pools hold free. The same before a buffer's first use and after its free,
// wherever the free has put it.
size_t dev_available(cudaStream_t s) {
  size_t free_b = 0, total_b = 0;
  EVOC_CUDA(cudaMemGetInfo(&free_b, &total_b));
  int device = 0;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_pools.find(s);
    if (it != g_pools.end()) device = it->second.device;
    for (auto& p : g_pools)
      if (p.second.device == device) free_b += p.second.bytes;
  }
  cudaMemPool_t pool;
  uint64_t reserved = 0, used = 0;
  if (cudaDeviceGetDefaultMemPool(&pool, device) == cudaSuccess &&
      cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved) == cudaSuccess &&
      cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) == cudaSuccess &&
      reserved > used)
    free_b += reserved - used;
  (void)cudaGetLastError();
  return free_b;
}

// A buffer of at least `bytes`; *held is its size class, to be given to dev_free.
cudaError_t dev_alloc(void** ptr, size_t bytes, cudaStream_t s, size_t* held) {
  const size_t cls = class_of(bytes);
  {
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_pools.find(s);
    if (it != g_pools.end() && (*ptr = it->second.take(cls, held))) return cudaSuccess;
  }
  *held = cls;
  cudaError_t e = cudaMallocAsync(ptr, cls, s);
  if (e == cudaSuccess) return e;
  (void)cudaGetLastError();
  int device = -1;
  {  // give back what this stream holds
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_pools.find(s);
    if (it != g_pools.end()) {
      it->second.shrink(0, s);
      device = it->second.device;
    }
  }
  e = cudaMallocAsync(ptr, cls, s);
  if (e == cudaSuccess) return e;
  (void)cudaGetLastError();
  {  // then what the others on the device do, once their streams are done with it
    std::lock_guard<std::mutex> lk(g_mu);
    for (auto& p : g_pools) {
      if (p.first == s || p.second.device != device || p.second.capturing || !p.second.bytes)
        continue;
      cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;  // by the caller's own hand
      if (cudaStreamIsCapturing(p.first, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
        (void)cudaGetLastError();
        continue;
      }
      p.second.shrink(0, p.first);
      cudaStreamSynchronize(p.first);
    }
  }
  return cudaMallocAsync(ptr, cls, s);
}

void dev_free(void* ptr, size_t held, cudaStream_t s) {
  {
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_pools.find(s);
    if (it != g_pools.end() && held <= it->second.limit) {
      Pool& p = it->second;
      p.shrink(p.limit - held, s);
      try {
        p.free_blocks[held].push_back(Block{ptr, ++p.stamp});
        p.bytes += held;
        return;
      } catch (const std::bad_alloc&) {  // no host memory for the entry: not kept
      }
    }
  }
  cudaFreeAsync(ptr, s);
}

}  // namespace evoc
