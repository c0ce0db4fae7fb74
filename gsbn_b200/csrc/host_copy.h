/*
 * host_copy.h -- device-to-host copies into the caller's pageable memory.
 *
 * A copy into pageable memory goes through the driver's own staging, one
 * thread at a time, at 4-8 GB/s into fresh pages, against 50 GB/s over the bus
 * into page-locked memory.  Large reads go through two page-locked chunks
 * instead: while one is filled, a few threads copy the other out, which also
 * spreads the first touch of the destination's pages.  The chunks are shared
 * by the process, allocated by a read that is worth it (kOwn) and freed with the
 * last handle (Users); a second reader at the same time, or one without memory
 * for them, takes the plain copy.
 */
#ifndef GSBN_HOST_COPY_H
#define GSBN_HOST_COPY_H

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>
#include <system_error>
#include <thread>
#include <vector>

namespace host_copy {

/* Plain / this way, in ms, on a 16-core host: into memory that the process has
   touched before 6 MB 0.57 / 0.39, 12 MB 1.14 / 0.72, 24 MB 2.2 / 1.1 (two
   threads, chunks of 4 MB); into fresh pages 32 MB 15 / 3.3, 40 MB 19 / 4.3, 64
   MB 30 / 6.2 (six threads, chunks of 8 MB).  Starting threads and first touches
   of the same huge page by several of them cost more than they give below. */
constexpr size_t kLeast = (size_t)6 << 20, kLarge = (size_t)24 << 20;
constexpr size_t kChunk = (size_t)8 << 20;

/* Allocating the two chunks takes 6 to 20 ms: as much as one copy of kOwn bytes
   gains (the first read of 32 MB 15.0 ms with the allocation, 15.1 plain; of 40
   MB 17.0, 18.8), but ten times what one of 8 MB does (18.7 ms with it, 0.8
   plain).  So a read of fewer bytes takes the plain copy until such reads have
   come to kSaved bytes since the chunks were last freed, and have lost by then
   about what the chunks cost. */
constexpr size_t kOwn = (size_t)32 << 20, kSaved = (size_t)192 << 20;

struct Shared {
  std::mutex use;   /* held during a copy */
  std::mutex count; /* everything below */
  int users = 0;
  void* chunk[2] = {nullptr, nullptr};
  size_t plain_bytes = 0;      /* large reads by the plain copy since the chunks were last freed */
  std::vector<void*> small;    /* free small buffers */
  std::vector<void*> pageable; /* small buffers, in use, of ordinary memory */
};

inline Shared& shared() {
  static Shared s;
  return s;
}

/* one per handle that may copy: the last one frees the chunks */
struct Users {
  Users() {
    std::lock_guard<std::mutex> l(shared().count);
    shared().users++;
  }
  ~Users() {
    Shared& s = shared();
    std::lock_guard<std::mutex> l(s.count);
    if (--s.users == 0) {
      for (void*& c : s.chunk) {
        if (c) cudaFreeHost(c);
        c = nullptr;
      }
      s.plain_bytes = 0;
    }
  }
  Users(const Users&) = delete;
  Users& operator=(const Users&) = delete;
};

/* a buffer of kSmall bytes for a handle's small results, page-locked where there
   is memory for that.  An allocation takes 1 to 3 ms, which a program that makes
   one network after the other would pay for each of them: so up to kSmallKept
   buffers (512 KB) stay for the process's next handles, past the last one.  One
   that a reset of the device has taken away is not handed out again: it is no
   longer page-locked or, if its address is another buffer's by now, without the
   mark it was left with. */
constexpr size_t kSmall = 65536, kSmallKept = 8;

struct Mark {
  uint64_t words[2];
  explicit Mark(const void* p) : words{0x6273676e5f6b6570ull, (uint64_t)(uintptr_t)p * 0x9e3779b97f4a7c15ull} {}
};

inline bool page_locked(const void* p) {
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, p) == cudaSuccess) return at.type == cudaMemoryTypeHost;
  cudaGetLastError();
  return false;
}

inline bool still_ours(const void* p) {
  const Mark m(p);
  return page_locked(p) && std::memcmp(p, &m, sizeof(m)) == 0;
}

inline void* take_small() {
  Shared& s = shared();
  std::lock_guard<std::mutex> l(s.count);
  while (!s.small.empty()) {
    void* p = s.small.back();
    s.small.pop_back();
    if (still_ours(p)) return p;
  }
  void* p = nullptr;
  if (cudaHostAlloc(&p, kSmall, cudaHostAllocPortable) == cudaSuccess) return p;
  cudaGetLastError(); /* ordinary memory serves: the copies into it are staged by the driver */
  try {
    s.pageable.reserve(s.pageable.size() + 1);
  } catch (const std::bad_alloc&) {
    return nullptr;
  }
  if ((p = std::malloc(kSmall))) s.pageable.push_back(p);
  return p;
}

inline void give_small(void* p) {
  if (!p) return;
  Shared& s = shared();
  std::lock_guard<std::mutex> l(s.count);
  const auto at = std::find(s.pageable.begin(), s.pageable.end(), p);
  if (at != s.pageable.end()) {
    s.pageable.erase(at);
    std::free(p);
    return;
  }
  if (!page_locked(p)) return; /* gone with a reset of the device */
  if (s.small.size() < kSmallKept) {
    try {
      s.small.push_back(p);
      const Mark m(p);
      std::memcpy(p, &m, sizeof(m));
      return;
    } catch (const std::bad_alloc&) {
    }
  }
  cudaFreeHost(p);
}

/* the chunks, for a read of `bytes`: there, or worth allocating for it */
inline bool chunks_ready(Shared& s, size_t bytes) {
  std::lock_guard<std::mutex> l(s.count);
  if (!(s.chunk[0] && s.chunk[1]) && bytes < kOwn) {
    s.plain_bytes += bytes;
    if (s.plain_bytes <= kSaved) return false;
  }
  for (void*& c : s.chunk)
    if (!c && cudaHostAlloc(&c, kChunk, cudaHostAllocPortable) != cudaSuccess) {
      c = nullptr;
      cudaGetLastError(); /* the plain copy needs none */
      return false;
    }
  return true;
}

inline cudaError_t plain(void* dst, const void* src, size_t bytes, cudaStream_t stream) {
  cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, stream);
  return e == cudaSuccess ? cudaStreamSynchronize(stream) : e;
}

/* copy on `stream` after the work queued there; complete on return */
inline cudaError_t to_host(void* dst, const void* src, size_t bytes, cudaStream_t stream) {
  if (bytes < kLeast) return plain(dst, src, bytes, stream);
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, dst) != cudaSuccess) cudaGetLastError();
  else if (at.type != cudaMemoryTypeUnregistered) return plain(dst, src, bytes, stream);
  Shared& s = shared();
  std::unique_lock<std::mutex> use(s.use, std::try_to_lock);
  if (!use.owns_lock() || !chunks_ready(s, bytes)) return plain(dst, src, bytes, stream);
  cudaEvent_t ev[3] = {nullptr, nullptr, nullptr}; /* of the chunks, and of the work queued before */
  for (cudaEvent_t& x : ev)
    if (cudaEventCreateWithFlags(&x, cudaEventDisableTiming) != cudaSuccess) {
      cudaGetLastError();
      for (cudaEvent_t y : ev)
        if (y) cudaEventDestroy(y);
      return plain(dst, src, bytes, stream);
    }
  const size_t chunk = bytes < kLarge ? kChunk / 2 : kChunk, n = (bytes + chunk - 1) / chunk;
  auto size = [&](size_t k) { return std::min(chunk, bytes - k * chunk); };
  auto post = [&](size_t k) {
    cudaError_t e = cudaMemcpyAsync(s.chunk[k & 1], (const uint8_t*)src + k * chunk, size(k), cudaMemcpyDeviceToHost, stream);
    return e == cudaSuccess ? cudaEventRecord(ev[k & 1], stream) : e;
  };
  /* chunks that are in, pieces of the copies out that are done; every thread
     copies its piece of every chunk */
  std::atomic<size_t> in{0}, out{0};
  std::atomic<bool> stop{false};
  int parts = 1;
  auto piece = [&](size_t k, int p) {
    const size_t len = size(k), step = ((len + parts - 1) / parts + 63) & ~(size_t)63, from = std::min(len, step * (size_t)p);
    std::memcpy((uint8_t*)dst + k * chunk + from, (const uint8_t*)s.chunk[k & 1] + from, std::min(step, len - from));
    out.fetch_add(1, std::memory_order_release);
  };
  auto work = [&](int p) {
    for (size_t k = 0; k < n; ++k) {
      while (in.load(std::memory_order_acquire) <= k) {
        if (stop.load(std::memory_order_relaxed)) return;
        std::this_thread::yield();
      }
      piece(k, p);
    }
  };
  cudaError_t e = cudaEventRecord(ev[2], stream);
  if (e == cudaSuccess) e = post(0);
  if (e == cudaSuccess && n > 1) e = post(1);
  /* the work queued before may take long: the others start after it, and spin for a chunk's copy at most */
  if (e == cudaSuccess) e = cudaEventSynchronize(ev[2]);
  std::vector<std::thread> team;
  const int want = (int)std::min(bytes < kLarge ? 2u : 6u, std::max(1u, std::thread::hardware_concurrency()));
  try {
    team.reserve(want - 1);
    parts = want; /* the pieces are fixed before the first thread copies: no chunk is in yet */
    for (int p = 1; p < want; ++p) team.emplace_back(work, p);
  } catch (const std::system_error&) {
    /* fewer threads than pieces: this thread copies the missing ones too */
  } catch (const std::bad_alloc&) {
  }
  const int have = (int)team.size() + 1;
  for (size_t k = 0; k < n && e == cudaSuccess; ++k) {
    e = cudaEventSynchronize(ev[k & 1]);
    if (e != cudaSuccess) break;
    in.store(k + 1, std::memory_order_release);
    piece(k, 0);
    for (int p = have; p < parts; ++p) piece(k, p);
    while (out.load(std::memory_order_acquire) < (k + 1) * (size_t)parts) std::this_thread::yield();
    if (k + 2 < n) e = post(k + 2);
  }
  stop = true;
  for (std::thread& t : team) t.join();
  cudaError_t last = cudaStreamSynchronize(stream); /* leave no copy into the chunks in flight */
  for (cudaEvent_t x : ev) cudaEventDestroy(x);
  return e != cudaSuccess ? e : last;
}

}  // namespace host_copy

#endif /* GSBN_HOST_COPY_H */
