// staging.hpp -- pinned host memory for transfers, and device memory that is
// cheap to take and give back.
//
// A copy to or from pageable memory goes through the driver's own staging
// buffer, one chunk after the other on the calling thread (26 MB of pointwise
// values: 1.3 ms, 18 GB/s), and costs 10 us and more however small it is.  Small
// transfers use a block of pinned memory that a session holds; large ones go
// through 1 MB blocks (48 GB/s; 41 at 512 KB), each copied by the copy engine
// while host threads move the blocks before it.
//
// Pinned and device allocations cost 1 to 5 ms and 40 to 150 us a call, more
// than a short run, so both come from process-wide pools that keep what is
// given back: 2 MB of small blocks, 8 MB of large ones and 96 MB of device
// memory at most, until the process ends.  Demand beyond that falls back to the
// driver.  Every function here is safe to call from several threads.
#pragma once
#include <cuda_runtime.h>
#include <emmintrin.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <map>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace gpum {

constexpr size_t kSmallPinned = 128 << 10;  // a session's block
constexpr size_t kSmallIn = 64 << 10;       // of it, for the host's inputs
constexpr size_t kSmallOut = kSmallPinned - kSmallIn;
constexpr size_t kChunkPinned = 1 << 20;    // a block of a large transfer
constexpr size_t kThreadedCopy = 4 * kChunkPinned;  // transfers moved by several threads
constexpr int kSmallBlocks = 16, kChunkBlocks = 8;

// One pinned allocation, made at the first use, in equal blocks.
class PinnedBlocks {
 public:
  PinnedBlocks(size_t block, int n) : block_(block), n_(n) {}
  // A block, or nullptr when all are taken (or there is no pinned memory).
  char* take() {
    std::lock_guard<std::mutex> lk(mu_);
    if (!tried_) {
      tried_ = true;
      void* p = nullptr;
      if (cudaHostAlloc(&p, block_ * n_, cudaHostAllocPortable) == cudaSuccess) {
        for (int i = 0; i < n_; ++i) free_.push_back(static_cast<char*>(p) + i * block_);
      } else {
        cudaGetLastError();
      }
    }
    if (free_.empty()) return nullptr;
    char* p = free_.back();
    free_.pop_back();
    return p;
  }
  // The caller has waited for every transfer that used the block.
  void give(char* p) {
    if (!p) return;
    std::lock_guard<std::mutex> lk(mu_);
    free_.push_back(p);
  }

 private:
  const size_t block_;
  const int n_;
  std::mutex mu_;
  bool tried_ = false;
  std::vector<char*> free_;
};

// Never destroyed, so that they outlive every session; inline functions, so
// that the library has one of each.
inline PinnedBlocks& pinned_small() {
  static PinnedBlocks* p = new PinnedBlocks(kSmallPinned, kSmallBlocks);
  return *p;
}
inline PinnedBlocks& pinned_chunks() {
  static PinnedBlocks* p = new PinnedBlocks(kChunkPinned, kChunkBlocks);
  return *p;
}

// ------------------------------------------------------------ device memory
// Allocations up to kPoolMax come from a memory pool of the current device
// that keeps at most kPoolKeep when nothing is allocated.  As with cudaMalloc
// the memory is usable on every stream at once.  It goes back to the pool and
// device that it came from, whatever device is current: on the pool's stream when
// its owner's stream is idle, so that the next allocation may take it at once,
// else on its owner's, and the pool hands it out again when that is done.
// Nothing here waits for a device: another thread may be capturing a graph, and
// CUDA allows no such wait meanwhile.
// 96 MB hold three sessions of 65,537 x 17 values, packed copy and partial sums
// included; with 64 MB a new one's first gradient call allocated anew (500 us,
// 200 without).
constexpr size_t kPoolMax = 32u << 20;
constexpr uint64_t kPoolKeep = 96ull << 20;

struct DevicePool {
  cudaMemPool_t pool = nullptr;
  cudaStream_t st = nullptr;
  int dev = -1;
};
inline DevicePool* device_pool() {
  static std::mutex* mu = new std::mutex();
  static std::map<int, DevicePool>* pools = new std::map<int, DevicePool>();
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
  std::lock_guard<std::mutex> lk(*mu);
  auto it = pools->find(dev);
  if (it == pools->end()) {
    DevicePool d;
    d.dev = dev;
    cudaMemPoolProps pp{};
    pp.allocType = cudaMemAllocationTypePinned;
    pp.location.type = cudaMemLocationTypeDevice;
    pp.location.id = dev;
    uint64_t keep = kPoolKeep;
    int wait = 0;  // an allocation does not queue behind other owners' work
    if (cudaMemPoolCreate(&d.pool, &pp) != cudaSuccess ||
        cudaMemPoolSetAttribute(d.pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess ||
        cudaMemPoolSetAttribute(d.pool, cudaMemPoolReuseAllowInternalDependencies, &wait) !=
            cudaSuccess ||
        cudaStreamCreateWithFlags(&d.st, cudaStreamNonBlocking) != cudaSuccess) {
      cudaGetLastError();
      d = DevicePool{};  // plain allocations on this device
    }
    it = pools->emplace(dev, d).first;
  }
  return it->second.pool ? &it->second : nullptr;
}

// An allocation, and where it goes back.
struct DevMem {
  void* p = nullptr;
  DevicePool* pool = nullptr;  // that it came from; nullptr: plain
  cudaStream_t st = nullptr;   // the owner's stream
};
// For the owner of stream `st`, which outlives the allocation.
inline cudaError_t dev_alloc(DevMem* m, size_t bytes, cudaStream_t st) {
  *m = DevMem{};
  m->st = st;
  DevicePool* d = device_pool();
  if (!d || bytes > kPoolMax) {
    cudaError_t e = cudaMalloc(&m->p, bytes);
    if (e == cudaErrorMemoryAllocation && d && cudaMemPoolTrimTo(d->pool, 0) == cudaSuccess) {
      cudaGetLastError();
      e = cudaMalloc(&m->p, bytes);  // with what the pool kept
    }
    return e;
  }
  m->pool = d;
  cudaError_t e = cudaMallocFromPoolAsync(&m->p, bytes, d->pool, d->st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(d->st);
  return e;
}
inline void dev_free(DevMem* m) {
  if (!m->p) return;
  if (!m->pool) {
    cudaFree(m->p);  // which waits for its device
  } else {
    int dev = m->pool->dev;
    cudaGetDevice(&dev);
    if (dev != m->pool->dev) cudaSetDevice(m->pool->dev);
    const bool idle = cudaStreamQuery(m->st) == cudaSuccess;
    if (cudaFreeAsync(m->p, idle ? m->pool->st : m->st) != cudaSuccess) {
      // Without a stream's order: after a wait for the owner's, or, if that fails
      // too (the context is lost), not at all.
      if (cudaStreamSynchronize(m->st) == cudaSuccess) cudaFree(m->p);
    }
    cudaGetLastError();
    if (dev != m->pool->dev) cudaSetDevice(dev);
  }
  *m = DevMem{};
}

// A stream that outlives the buffers declared after it.
struct OwnedStream {
  cudaStream_t s = nullptr;
  OwnedStream() = default;
  OwnedStream(const OwnedStream&) = delete;
  OwnedStream& operator=(const OwnedStream&) = delete;
  ~OwnedStream() {
    if (s) cudaStreamDestroy(s);
  }
};

// Waits for a stream on the way out, errors included: where work on it uses
// memory of another owner, who may give it back next.
struct WaitAtExit {
  cudaStream_t st;
  ~WaitAtExit() { cudaStreamSynchronize(st); }
};

// ---------------------------------------------------------- large transfers
inline void convert_copy(float* dst, const float* src, size_t n) {
  std::memcpy(dst, src, n * sizeof(float));
}
inline void convert_copy(double* dst, const double* src, size_t n) {
  std::memcpy(dst, src, n * sizeof(double));
}
// f32 to f64, with stores that do not read the destination's lines first
// (64 MB on six threads: 0.76 ms, with plain stores 1.46).
inline void convert_copy(double* dst, const float* src, size_t n) {
  size_t k = 0;
  if (n > 0 && (reinterpret_cast<uintptr_t>(dst) & 15)) dst[k] = (double)src[k], ++k;
  for (; k + 4 <= n; k += 4) {
    const __m128 v = _mm_loadu_ps(src + k);
    _mm_stream_pd(dst + k, _mm_cvtps_pd(v));
    _mm_stream_pd(dst + k + 2, _mm_cvtps_pd(_mm_movehl_ps(v, v)));
  }
  for (; k < n; ++k) dst[k] = (double)src[k];
  _mm_sfence();
}

// n device values into pageable host memory after the work already enqueued
// on `st` (f32 values may widen to f64 on the way, which is exact); returns
// when they have arrived.  The calling thread keeps a ring of pinned blocks
// filled by the copy engine.  Below 4 MB it moves them on itself, in pieces of
// 512 KB (1.5 MB widened to 3: 143 us; 1 MB pieces and two threads, whose start
// takes as long as the copy, 290; the driver's staging of the 3 MB 187).  Above,
// it hands blocks of 1 MB to up to five threads (4 MB to 8: 261 us, alone 360;
// 13 MB to 26: 0.53 to 0.67 ms, alone 1.25, the driver 1.33; threads that each
// copied and moved their own blocks 0.75 to 1.5).
template <class To, class From>
cudaError_t copy_to_host(To* dst, const From* src, size_t n, cudaStream_t st) {
  // The threads poll for chunks, so they start when there is something to copy.
  cudaError_t e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return e;
  const bool alone = n * sizeof(From) < kThreadedCopy;
  const size_t per = (alone ? kChunkPinned / 2 : kChunkPinned) / sizeof(From);
  const size_t chunks = (n + per - 1) / per;
  const size_t want = std::min<size_t>(kChunkBlocks, std::max<size_t>(chunks, 1));
  std::vector<char*> blocks;
  std::vector<cudaEvent_t> ev;
  while (blocks.size() < want) {
    char* p = pinned_chunks().take();
    if (!p) break;
    blocks.push_back(p);
    cudaEvent_t v = nullptr;
    e = cudaEventCreateWithFlags(&v, cudaEventDisableTiming);
    if (e != cudaSuccess) break;
    ev.push_back(v);
  }
  if (blocks.empty()) {  // all taken: the driver's staging
    std::vector<From> tmp(n);
    e = cudaMemcpyAsync(tmp.data(), src, n * sizeof(From), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess) convert_copy(dst, tmp.data(), n);
    return e;
  }
  const size_t nb = ev.size();
  // ready: chunks that have arrived (or SIZE_MAX: give up); moved[b]: chunks of
  // block b that have been moved on.
  std::atomic<size_t> ready{0}, next{0};
  std::vector<std::atomic<size_t>> moved(blocks.size());
  for (auto& m : moved) m.store(0);
  auto move = [&](size_t k) {
    const size_t at = k * per;
    convert_copy(dst + at, reinterpret_cast<const From*>(blocks[k % nb]), std::min(per, n - at));
    moved[k % nb].fetch_add(1, std::memory_order_release);
  };
  auto work = [&] {
    for (size_t k; (k = next.fetch_add(1)) < chunks;) {
      size_t r;
      while ((r = ready.load(std::memory_order_acquire)) <= k) _mm_pause();
      if (r == SIZE_MAX) return;
      move(k);
    }
  };
  std::vector<std::thread> threads;
  if (e == cudaSuccess && !alone) {
    const size_t cores = std::max(1u, std::thread::hardware_concurrency() / 2);
    const size_t nt = std::min<size_t>(std::min<size_t>(5, cores), chunks);
    threads.reserve(nt);
    for (size_t i = 0; i < nt; ++i) {
      try {
        threads.emplace_back(work);
      } catch (const std::system_error&) {
        break;  // no more threads: the ones that run (or the caller) do it
      }
    }
  }
  size_t sent = 0, here = 0;
  while (e == cudaSuccess && here < chunks) {
    while (e == cudaSuccess && sent < chunks &&
           moved[sent % nb].load(std::memory_order_acquire) >= sent / nb) {
      const size_t at = sent * per;
      e = cudaMemcpyAsync(blocks[sent % nb], src + at, std::min(per, n - at) * sizeof(From),
                          cudaMemcpyDeviceToHost, st);
      if (e == cudaSuccess) e = cudaEventRecord(ev[sent % nb], st);
      ++sent;
    }
    if (e != cudaSuccess || here == sent) continue;
    e = cudaEventQuery(ev[here % nb]);
    if (e == cudaSuccess) {
      if (threads.empty()) move(here);
      ready.store(++here, std::memory_order_release);
    } else if (e == cudaErrorNotReady) {
      e = cudaSuccess;
    }
  }
  if (e != cudaSuccess) {
    ready.store(SIZE_MAX, std::memory_order_release);
    cudaStreamSynchronize(st);  // no copy into a block is left
  }
  for (std::thread& t : threads) t.join();
  for (cudaEvent_t v : ev) cudaEventDestroy(v);
  for (char* p : blocks) pinned_chunks().give(p);
  return e;
}

// Whether a host pointer is pinned, so that a plain copy runs at full speed.
inline bool host_is_pinned(const void* p) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeHost || a.type == cudaMemoryTypeManaged;
}

}  // namespace gpum
