// host_staging.h -- large copies between pageable host memory and the device
// through two pinned 64 MiB chunks: the DMA of one chunk overlaps the copy of
// the other between pinned and pageable memory, which runs on all OpenMP
// threads (so first touch of fresh pageable pages is parallel too).  Used by
// the mesh set-up paths, whose arrays reach several GB.
#ifndef CGX_HOST_STAGING_H
#define CGX_HOST_STAGING_H

#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstring>
#include <map>
#include <mutex>
#include <vector>

namespace cgx_staging {

inline void par_memcpy(void* dst, const void* src, size_t bytes) {
  const size_t blk = size_t(1) << 20;
  const long long nb = (long long)((bytes + blk - 1) / blk);
#pragma omp parallel for schedule(static)
  for (long long b = 0; b < nb; ++b) {
    const size_t off = size_t(b) * blk;
    std::memcpy(static_cast<char*>(dst) + off, static_cast<const char*>(src) + off, std::min(blk, bytes - off));
  }
}

constexpr size_t kChunk = size_t(64) << 20;

// The two pinned chunks of a Staging and the events of their last copies.
// Page-locking 128 MiB takes 60 to 100 ms, most of the set-up of a small mesh
// and of a solver's first pageable copy, so chunks that were given back are
// kept for the next user of their device: at most as many pairs as the device has
// registered users (solvers that have staged a copy), and kKept where there are
// fewer.  So threads that copy together, each for its own solver, page-lock once
// and not in every round of calls, no more is held than a pair per solver, and
// what is kept when the solvers are gone is kKept pairs.  A pair belongs to one
// Staging at a time and comes back idle (its stream synchronised); the lists are
// guarded for use from several threads, and pairs are released outside the lock.
// Four threads that set and get the state of 195,000 cells each: 2.5 ms a round of
// calls (150 ms with two kept pairs in all, 2.3 ms with a pair held per solver).
struct Chunks {
  int device = -1;
  char* pin[2] = {nullptr, nullptr};
  cudaEvent_t done[2] = {nullptr, nullptr};

  void free_all() {
    for (int i = 0; i < 2; ++i) {
      if (pin[i]) cudaFreeHost(pin[i]);
      if (done[i]) cudaEventDestroy(done[i]);
    }
  }
};

constexpr size_t kKept = 2;
struct ChunkPool {
  std::mutex mu;
  std::vector<Chunks> idle;
  std::map<int, size_t> users;  // per device

  size_t idle_of(int device) const {
    size_t n = 0;
    for (const Chunks& c : idle) n += (c.device == device);
    return n;
  }
  size_t limit(int device) const {
    const auto u = users.find(device);
    return std::max(kKept, u == users.end() ? size_t(0) : u->second);
  }
};
inline ChunkPool& chunk_pool() {
  static ChunkPool* p = new ChunkPool();  // outlives every static user
  return *p;
}

// a pair for the current device: a kept one that is still valid (a reset of
// the device takes it away), or a new one
inline cudaError_t take_chunks(Chunks* c) {
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  {
    ChunkPool& p = chunk_pool();
    std::lock_guard<std::mutex> lk(p.mu);
    for (size_t i = p.idle.size(); i-- > 0;) {
      if (p.idle[i].device != device) continue;
      Chunks k = p.idle[i];
      p.idle.erase(p.idle.begin() + long(i));
      cudaPointerAttributes a0{}, a1{};
      if (cudaPointerGetAttributes(&a0, k.pin[0]) == cudaSuccess && a0.type == cudaMemoryTypeHost &&
          cudaPointerGetAttributes(&a1, k.pin[1]) == cudaSuccess && a1.type == cudaMemoryTypeHost) {
        *c = k;
        return cudaSuccess;
      }
      cudaGetLastError();  // gone with its context
    }
  }
  c->device = device;
  for (int i = 0; i < 2 && e == cudaSuccess; ++i) {
    e = cudaMallocHost(reinterpret_cast<void**>(&c->pin[i]), kChunk);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&c->done[i], cudaEventDisableTiming);
  }
  return e;
}

inline void give_back(const Chunks& c) {
  ChunkPool& p = chunk_pool();
  {
    std::lock_guard<std::mutex> lk(p.mu);
    if (c.pin[0] && c.pin[1] && c.done[0] && c.done[1] && p.idle_of(c.device) < p.limit(c.device)) {
      p.idle.push_back(c);
      return;
    }
  }
  Chunks k = c;
  k.free_all();
}

// A registered user of a device's chunks, for as long as it lives.
class User {
 public:
  explicit User(int device) : device_(device) {
    ChunkPool& p = chunk_pool();
    std::lock_guard<std::mutex> lk(p.mu);
    ++p.users[device_];
  }
  User(const User&) = delete;
  User& operator=(const User&) = delete;
  ~User() {
    ChunkPool& p = chunk_pool();
    std::vector<Chunks> over;
    {
      std::lock_guard<std::mutex> lk(p.mu);
      --p.users[device_];
      size_t n = p.idle_of(device_);
      for (size_t i = p.idle.size(); i-- > 0 && n > p.limit(device_);)
        if (p.idle[i].device == device_) {
          over.push_back(p.idle[i]);
          p.idle.erase(p.idle.begin() + long(i));
          --n;
        }
    }
    for (Chunks& c : over) c.free_all();
  }

 private:
  int device_;
};

class Staging {
 public:
  explicit Staging(cudaStream_t s) : s_(s) {}
  Staging(const Staging&) = delete;
  Staging& operator=(const Staging&) = delete;

  // pinned buffers and events; must succeed before put/get
  cudaError_t init() { return take_chunks(&c_); }

  ~Staging() {
    // no DMA may still target the buffers; if that cannot be known, they stay
    // with the process
    if (cudaStreamSynchronize(s_) == cudaSuccess) give_back(c_);
  }

  // host -> device, asynchronous on the stream (src may be reused on return)
  cudaError_t put(void* dst, const void* src, size_t bytes) {
    const size_t nch = (bytes + kChunk - 1) / kChunk;
    for (size_t c = 0; c < nch; ++c) {
      const size_t off = c * kChunk, len = std::min(kChunk, bytes - off);
      cudaError_t e = cudaEventSynchronize(c_.done[c & 1]);  // the buffer's previous DMA
      if (e != cudaSuccess) return e;
      par_memcpy(c_.pin[c & 1], static_cast<const char*>(src) + off, len);
      e = cudaMemcpyAsync(static_cast<char*>(dst) + off, c_.pin[c & 1], len, cudaMemcpyHostToDevice, s_);
      if (e != cudaSuccess) return e;
      e = cudaEventRecord(c_.done[c & 1], s_);
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  }

  // device -> host, complete on return; on `st` instead of the object's
  // stream when given (the copies then follow st's earlier work)
  cudaError_t get(void* dst, const void* src, size_t bytes, cudaStream_t st = nullptr) {
    cudaStream_t q = st ? st : s_;
    const cudaError_t e = get_on(q, dst, src, bytes);
    if (e != cudaSuccess) cudaStreamSynchronize(q);  // leave no copy in flight behind an error
    return e;
  }

 private:
  cudaError_t get_on(cudaStream_t q, void* dst, const void* src, size_t bytes) {
    const size_t nch = (bytes + kChunk - 1) / kChunk;
    for (size_t c = 0; c < nch; ++c) {
      const size_t off = c * kChunk, len = std::min(kChunk, bytes - off);
      cudaError_t e = cudaMemcpyAsync(c_.pin[c & 1], static_cast<const char*>(src) + off, len,
                                      cudaMemcpyDeviceToHost, q);
      if (e != cudaSuccess) return e;
      e = cudaEventRecord(c_.done[c & 1], q);
      if (e != cudaSuccess) return e;
      if (c > 0 && (e = drain(static_cast<char*>(dst), c - 1, bytes)) != cudaSuccess) return e;
    }
    return nch > 0 ? drain(static_cast<char*>(dst), nch - 1, bytes) : cudaSuccess;
  }

  cudaError_t drain(char* dst, size_t c, size_t bytes) {
    const size_t off = c * kChunk, len = std::min(kChunk, bytes - off);
    const cudaError_t e = cudaEventSynchronize(c_.done[c & 1]);
    if (e != cudaSuccess) return e;
    par_memcpy(dst + off, c_.pin[c & 1], len);
    return cudaSuccess;
  }

  cudaStream_t s_;
  Chunks c_;
};

}  // namespace cgx_staging

#endif
