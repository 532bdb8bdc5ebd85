// host_pool.h - page-locked host memory handed to callers (freed with cuda_free_host).
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <chrono>
#include <cstddef>
#include <cstdint>
#include <condition_variable>
#include <cstring>
#include <iterator>
#include <map>
#include <mutex>
#include <thread>
#include <unordered_map>
#include <vector>

namespace crb {

static inline size_t pool_round_up(size_t x, size_t q) { return (x + q - 1) / q * q; }

// Results are handed to the caller in page-locked memory that it frees with cuda_free_host.
// Pinning fresh memory for every result costs far more than the copy itself, so freed
// blocks are kept (up to kMaxIdle bytes) and reused for later results of similar size.
class PinnedPool {
 public:
  void* get(size_t n, cudaError_t* err) {
    const size_t want = pool_round_up(n ? n : 1, 64 << 10);
    {
      std::lock_guard<std::mutex> g(mu_);
      auto it = idle_.lower_bound(want);
      // (a request of a few bytes takes no large block from the transfers: pinning that anew costs far more)
      const size_t slack = want <= kSmall ? want : want / 2 + (64ull << 20);
      if (it != idle_.end() && it->first <= want + slack) {
        void* p = it->second.first;
        idle_bytes_ -= it->first;
        lru_.erase(it->second.second);
        idle_.erase(it);
        *err = cudaSuccess;
        return p;
      }
    }
    void* p = nullptr;
    *err = cudaMallocHost(&p, want);
    if (*err != cudaSuccess) return nullptr;
    std::lock_guard<std::mutex> g(mu_);
    sizes_[p] = want;
    return p;
  }
  // Keep p for reuse. Over kMaxIdle idle bytes, the blocks idle the longest are released first
  // (so a large block handed back, the one most likely wanted again soon, is kept).
  void put(void* p) {
    if (!p) return;
    std::vector<void*> evict;
    {
      std::lock_guard<std::mutex> g(mu_);
      auto s = sizes_.find(p);
      if (s == sizes_.end()) {
        evict.push_back(p);  // not ours: release directly
      } else {
        const unsigned long long seq = ++seq_;
        idle_.emplace(s->second, std::make_pair(p, seq));
        lru_.emplace(seq, std::make_pair(s->second, p));
        idle_bytes_ += s->second;
        while (idle_bytes_ > kMaxIdle && !lru_.empty()) {
          auto old = lru_.begin();
          if (old->first == seq && lru_.size() > 1) old = std::next(old);  // not the block just returned
          const size_t sz = old->second.first;
          void* q = old->second.second;
          auto range = idle_.equal_range(sz);
          for (auto it = range.first; it != range.second; ++it)
            if (it->second.first == q) {
              idle_.erase(it);
              break;
            }
          idle_bytes_ -= sz;
          sizes_.erase(q);
          evict.push_back(q);
          lru_.erase(old);
        }
      }
    }
    for (void* q : evict) cudaFreeHost(q);
  }

 private:
  static constexpr size_t kMaxIdle = 24ull << 30;
  static constexpr size_t kSmall = 64u << 10;
  std::mutex mu_;
  std::multimap<size_t, std::pair<void*, unsigned long long>> idle_;  // size -> (block, put order)
  std::map<unsigned long long, std::pair<size_t, void*>> lru_;        // put order -> (size, block)
  std::unordered_map<void*, size_t> sizes_;
  size_t idle_bytes_ = 0;
  unsigned long long seq_ = 0;
};

// The process-wide pool (never destroyed: CUDA may be torn down first at exit).
PinnedPool& host_pinned_pool();

// A few persistent host threads for memcpys from 1 MiB (pageable <-> page-locked staging, result
// copies): spawning threads per copy would cost more than the copy of a staging piece. The parts of a copy are
// taken one by one, by the calling thread too; the workers help the oldest copy that has parts left, so copies of
// several threads run side by side (one at a time, with small ones left to their callers meanwhile, two sessions on 24 MiB documents
// took 3.2 ms a round, four 5.1; so 2.5 and 4.3). A worker looks out for the next copy for a moment before it sleeps, so the pieces of a
// pipelined transfer follow each other without a wake-up each.
class CopyWorkers {
 public:
  static constexpr size_t kMin = 1u << 20, kPart = 256u << 10;
  static CopyWorkers& get() {
    static CopyWorkers* w = new CopyWorkers();  // never destroyed (threads parked at exit)
    return *w;
  }
  // dst[0, n) = src[0, n), split across the workers and the calling thread
  void copy(void* dst, const void* src, size_t n) {
    if (n < kMin || nthreads_ == 0) {
      memcpy(dst, src, n);
      return;
    }
    Copy c;
    c.dst = static_cast<char*>(dst);
    c.src = static_cast<const char*>(src);
    c.n = n;
    const size_t most = n / kPart;
    c.parts = most < nthreads_ + 1u ? most : nthreads_ + 1u;
    c.part = pool_round_up((n + c.parts - 1) / c.parts, 4096);
    c.pending = c.parts;
    std::unique_lock<std::mutex> lk(mu_);
    (last_ ? last_->following : first_) = &c;
    last_ = &c;
    waiting_.fetch_add(1, std::memory_order_release);
    if (asleep_) work_.notify_all();
    while (c.next < c.parts) take_part(lk, c);
    done_.wait(lk, [&] { return c.pending == 0; });
  }

 private:
  struct Copy {  // lives on its caller's stack
    char* dst;
    const char* src;
    size_t n, part, parts, next = 0, pending;
    Copy* following = nullptr;
  };
  CopyWorkers() {
    const unsigned hw = std::thread::hardware_concurrency();
    nthreads_ = hw > 1 ? (hw - 1 < 15u ? hw - 1 : 15u) : 0u;
    for (unsigned i = 0; i < nthreads_; ++i) std::thread([this] { loop(); }).detach();
  }
  // one part of c, which has some left (lk held on entry and exit, not while copying)
  void take_part(std::unique_lock<std::mutex>& lk, Copy& c) {
    const size_t a = c.part * c.next++;
    const size_t len = a < c.n ? (c.part < c.n - a ? c.part : c.n - a) : 0;
    if (c.next == c.parts) {  // none left: out of the list
      Copy** at = &first_;
      Copy* before = nullptr;
      for (; *at != &c; at = &(*at)->following) before = *at;
      *at = c.following;
      if (last_ == &c) last_ = before;
      waiting_.fetch_sub(1, std::memory_order_relaxed);
    }
    char* d = c.dst;
    const char* f = c.src;
    lk.unlock();
    if (len) memcpy(d + a, f + a, len);
    lk.lock();
    if (--c.pending == 0) done_.notify_all();
  }
  void loop() {
    for (;;) {
      const auto until = std::chrono::steady_clock::now() + std::chrono::microseconds(60);
      while (!waiting_.load(std::memory_order_acquire) && std::chrono::steady_clock::now() < until) std::this_thread::yield();
      std::unique_lock<std::mutex> lk(mu_);
      ++asleep_;
      work_.wait(lk, [&] { return first_ != nullptr; });
      --asleep_;
      while (first_) take_part(lk, *first_);
    }
  }
  std::mutex mu_;
  std::condition_variable work_, done_;
  unsigned nthreads_ = 0, asleep_ = 0;
  Copy *first_ = nullptr, *last_ = nullptr;  // copies with parts left, the oldest first
  std::atomic<unsigned> waiting_{0};         // how many those are
};

// memcpy split over the copy workers when it is large.
inline void parallel_memcpy(void* dst, const void* src, size_t n) { CopyWorkers::get().copy(dst, src, n); }

// Copies ranges of page-locked host memory into pageable caller memory as their downloads
// land: push() queues (dst, src, n) behind an event recorded after the range's device-to-host
// copy; a thread of its own waits for each event in turn and copies the range on the copy
// workers, so the copy of one chunk's output overlaps the downloads and kernels of the next.
// The downloads themselves go at the link's rate into a page-locked block (a DMA into pageable
// memory is staged by the driver at a fraction of it). finish() waits for every queued range.
class CopyOut {
 public:
  void open(int device) {
    th_ = std::thread([this, device] { loop(device); });
  }
  void push(uint8_t* dst, const uint8_t* src, size_t n, cudaEvent_t ready) {
    if (!n) return;
    std::lock_guard<std::mutex> g(mu_);
    q_.push_back(Item{dst, src, n, ready});
    cv_.notify_all();
  }
  // waits for every queued range; the first error met (later ranges are skipped after one)
  cudaError_t finish() {
    {
      std::lock_guard<std::mutex> g(mu_);
      closed_ = true;
      cv_.notify_all();
    }
    if (th_.joinable()) th_.join();
    return err_;
  }
  ~CopyOut() { finish(); }

 private:
  struct Item {
    uint8_t* dst;
    const uint8_t* src;
    size_t n;
    cudaEvent_t ready;
  };
  void loop(int device) {
    if (cudaSetDevice(device) != cudaSuccess) err_ = cudaErrorInvalidDevice;
    for (;;) {
      Item it;
      {
        std::unique_lock<std::mutex> lk(mu_);
        cv_.wait(lk, [&] { return !q_.empty() || closed_; });
        if (q_.empty()) break;
        it = q_.front();
        q_.erase(q_.begin());
      }
      if (err_ != cudaSuccess) continue;
      if (it.ready) err_ = cudaEventSynchronize(it.ready);
      if (err_ == cudaSuccess) parallel_memcpy(it.dst, it.src, it.n);
    }
  }
  std::thread th_;
  std::mutex mu_;
  std::condition_variable cv_;
  std::vector<Item> q_;
  bool closed_ = false;
  cudaError_t err_ = cudaSuccess;  // written by the thread only until finish() joins it
};

// First-fit sub-allocator over one page-locked block: a server's host staging area, pinned
// once instead of per request. Blocks handed to callers are released with cuda_free_host
// (host_free below finds the owning area); an area closed by its server is freed when its
// last block comes back.
class HostArena {
 public:
  ~HostArena() {
    if (base_) cudaFreeHost(base_);
  }
  cudaError_t init(size_t bytes) {
    bytes = pool_round_up(bytes ? bytes : 1, 2u << 20);
    cudaError_t e = cudaMallocHost(&base_, bytes);
    if (e != cudaSuccess) {
      base_ = nullptr;
      return e;
    }
    size_ = bytes;
    free_[0] = bytes;
    return cudaSuccess;
  }
  uint8_t* alloc(size_t n) {
    n = pool_round_up(n ? n : 1, 256);
    std::lock_guard<std::mutex> g(mu_);
    for (auto it = free_.begin(); it != free_.end(); ++it) {
      if (it->second >= n) {
        const size_t off = it->first, rest = it->second - n;
        free_.erase(it);
        if (rest) free_[off + n] = rest;
        used_[off] = n;
        return base_ + off;
      }
    }
    return nullptr;
  }
  bool contains(const void* p) const {
    const uint8_t* q = static_cast<const uint8_t*>(p);
    return base_ && q >= base_ && q < base_ + size_;
  }
  // returns true when the area is closed and now empty
  bool release(const void* p) {
    std::lock_guard<std::mutex> g(mu_);
    size_t start = (size_t)(static_cast<const uint8_t*>(p) - base_);
    auto u = used_.find(start);
    if (u == used_.end()) return false;
    size_t len = u->second;
    used_.erase(u);
    auto nx = free_.lower_bound(start);
    if (nx != free_.end() && start + len == nx->first) {
      len += nx->second;
      nx = free_.erase(nx);
    }
    if (nx != free_.begin()) {
      auto pv = std::prev(nx);
      if (pv->first + pv->second == start) {
        start = pv->first;
        len += pv->second;
        free_.erase(pv);
      }
    }
    free_[start] = len;
    return closed_ && used_.empty();
  }
  // the owner is gone; true when nothing is outstanding (the area can be freed now)
  bool close() {
    std::lock_guard<std::mutex> g(mu_);
    closed_ = true;
    return used_.empty();
  }

 private:
  std::mutex mu_;
  uint8_t* base_ = nullptr;
  size_t size_ = 0;
  bool closed_ = false;
  std::map<size_t, size_t> free_, used_;
};

// Registry of the live host areas (defined in capi.cu).
void host_arena_register(HostArena* a);
// The owner closes its area: freed now, or when its last block is released.
void host_arena_close(HostArena* a);
// Give the idle device blocks of finished streams back to the driver (stream.cu).
void dev_blocks_trim();
// cudaMalloc of this library: when memory has run out, the idle blocks go back and it is tried once more. An
// error is reported by the return value only (a later launch's cudaGetLastError does not see it).
cudaError_t dev_malloc_bytes(void** p, size_t n);
template <typename T>
cudaError_t dev_malloc(T** p, size_t n) {
  return dev_malloc_bytes(reinterpret_cast<void**>(p), n);
}
// Release a block handed to a caller: into its host area, else into the pool.
void host_free(void* p);

}  // namespace crb
