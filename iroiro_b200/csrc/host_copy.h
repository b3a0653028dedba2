// Copies between pageable host memory and a device through pinned slots.
//
// The driver copies pageable host memory through its own staging on one host
// thread, which also takes the page faults of a destination that was never
// touched (15.9 ms for the 75 MB force of a 16^3x32 lattice).  A larger copy is
// split into kRingSlot pieces that kCopyThreads host threads take in turn, each
// through two pinned slots of its own: its DMAs overlap its host copies and
// those of the other threads, and page faults are taken in parallel.  The slots
// (16 MB in all) are small so that the pipeline fills at once: with two 128 MB
// chunks the first DMA started after 4 ms of host copying.  Pinned memory,
// device-accessible memory and the copies that ring_pays() leaves out take the
// direct DMA.  The 75 MB force to the host 15.9 -> 2.1 ms; a 382 MB gauge
// upload 13.5 -> 9.6 ms.
//
// Only the CUDA runtime's C interface is used, so that a CPU test can link
// this against a runtime of its own.
#pragma once

#include <cuda_runtime_api.h>
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

namespace iro {

constexpr int kCopyThreads = 8;
constexpr size_t kRingSlot = size_t(1) << 20;

inline bool host_pageable(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

// Whether most of a destination's pages were never touched (no page is there
// yet): 16 of them are looked at.
inline bool host_untouched(const void* p, size_t bytes) {
  const uintptr_t page = uintptr_t(sysconf(_SC_PAGESIZE)), a = reinterpret_cast<uintptr_t>(p);
  int absent = 0;
  for (int k = 0; k < 16; ++k) {
    unsigned char v = 1;
    const uintptr_t q = (a + bytes / 16 * k + bytes / 32) / page * page;
    if (mincore(reinterpret_cast<void*>(q), page, &v) == 0 && !(v & 1)) ++absent;
  }
  return absent > 8;
}

// The copies that the slots make faster.  Starting the threads takes a
// hundred microseconds or two, which a copy has to win back.  Slots / direct,
// us (boxes differ by 10 %, by 25 % for the touched downloads):
//   upload, source in cache      4 MB 264 / 237, 8 MB 413 / 403, 10 MB 474 / 499, 16 MB 627 / 851
//   upload, source not in cache  4 MB 303 / 436, 8 MB 456 / 804, 10 MB 528 / 1011, 16 MB 686 / 1582
//   download, touched            8 MB 661 / 465, 16 MB 1073 / 870, 24 MB 1334 / 1391, 32 MB 1499 / 1678
//   download, untouched          4 MB 1175 / 1770, 16 MB 2655 / 7906, 64 MB 9264 / 32936
constexpr size_t kRingUp = size_t(10) << 20;
constexpr size_t kRingDown = size_t(32) << 20;
constexpr size_t kRingDownUntouched = size_t(4) << 20;
inline bool ring_pays(bool to_host, const void* host, size_t bytes) {
  if (!to_host) return bytes >= kRingUp;
  return bytes >= kRingDown || (bytes >= kRingDownUntouched && host_untouched(host, bytes));
}

// The slots of one device, shared by its contexts: allocated by the first copy
// that needs them, given back when the device's last context is destroyed.  One
// copy at a time uses them; another one that comes meanwhile (from another
// thread) takes the direct path.  The contexts' streams are not ordered among
// each other, so a copy ends, in either direction, only when its last DMAs have:
// no DMA needs a slot while `use` is free.
struct CopyRing {
  std::mutex use;
  char* buf = nullptr;
  cudaEvent_t ev[2 * kCopyThreads] = {};  // a slot's last DMA
  int contexts = 0;                       // guarded by ring_mutex()
};
constexpr int kRingDevices = 16;
inline CopyRing* ring_of(int device) {
  static CopyRing rings[kRingDevices];
  return device < 0 || device >= kRingDevices ? nullptr : &rings[device];
}
inline std::mutex& ring_mutex() {
  static std::mutex m;
  return m;
}

inline void ring_attach(int device) {
  CopyRing* r = ring_of(device);
  if (!r) return;
  std::lock_guard<std::mutex> lk(ring_mutex());
  ++r->contexts;
}
inline void ring_detach(int device) {
  CopyRing* r = ring_of(device);
  if (!r) return;
  std::lock_guard<std::mutex> lk(ring_mutex());
  if (--r->contexts > 0) return;
  if (r->buf) cudaFreeHost(r->buf);
  r->buf = nullptr;
  for (cudaEvent_t& e : r->ev) {
    if (e) cudaEventDestroy(e);
    e = nullptr;
  }
}

inline cudaError_t ensure_ring(CopyRing& r) {
  if (!r.buf) {
    const cudaError_t e =
        cudaHostAlloc(reinterpret_cast<void**>(&r.buf), 2 * kCopyThreads * kRingSlot, cudaHostAllocDefault);
    if (e != cudaSuccess) return e;
  }
  for (cudaEvent_t& v : r.ev)
    if (!v) {
      const cudaError_t e = cudaEventCreateWithFlags(&v, cudaEventDisableTiming);
      if (e != cudaSuccess) return e;
    }
  return cudaSuccess;
}

// One thread's share of a copy between `host` and `dev` through slots 2w and
// 2w + 1: pieces are taken from `next` until none is left, and the slots' last
// DMAs are waited for.  A slot's event marks its last DMA.
inline cudaError_t ring_worker(int device, cudaStream_t st, CopyRing& ring, int w, bool to_host, char* host, char* dev,
                               size_t bytes, std::atomic<size_t>& next) {
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) return e;
  char* slot[2] = {ring.buf + 2 * w * kRingSlot, ring.buf + (2 * w + 1) * kRingSlot};
  cudaEvent_t ev[2] = {ring.ev[2 * w], ring.ev[2 * w + 1]};
  const size_t none = ~size_t(0);
  size_t off[2] = {none, none};  // device to host: the piece in flight in each slot
  auto land = [&](int k) -> cudaError_t {
    if (off[k] == none) return cudaSuccess;
    const cudaError_t r = cudaEventSynchronize(ev[k]);
    if (r == cudaSuccess) std::memcpy(host + off[k], slot[k], std::min(kRingSlot, bytes - off[k]));
    off[k] = none;
    return r;
  };
  for (int k = 0;; k ^= 1) {
    if (to_host && (e = land(k)) != cudaSuccess) return e;
    const size_t o = next.fetch_add(1) * kRingSlot;
    if (o >= bytes) {
      if (to_host) return land(k ^ 1);
      e = cudaEventSynchronize(ev[k]);
      return e == cudaSuccess ? cudaEventSynchronize(ev[k ^ 1]) : e;
    }
    const size_t len = std::min(kRingSlot, bytes - o);
    if (to_host) {
      e = cudaMemcpyAsync(slot[k], dev + o, len, cudaMemcpyDeviceToHost, st);
      off[k] = o;
    } else {
      // the slot's previous DMA is done
      if ((e = cudaEventSynchronize(ev[k])) != cudaSuccess) return e;
      std::memcpy(slot[k], host + o, len);
      e = cudaMemcpyAsync(dev + o, slot[k], len, cudaMemcpyHostToDevice, st);
    }
    if (e == cudaSuccess) e = cudaEventRecord(ev[k], st);
    if (e != cudaSuccess) return e;
  }
}

inline cudaError_t ring_copy(int device, cudaStream_t st, CopyRing& ring, bool to_host, char* host, char* dev,
                             size_t bytes) {
  std::atomic<size_t> next{0};
  const int nt = int(std::min<size_t>(std::min<unsigned>(kCopyThreads, std::max(1u, std::thread::hardware_concurrency())),
                                      (bytes + kRingSlot - 1) / kRingSlot));
  cudaError_t err[kCopyThreads] = {};
  std::vector<std::thread> th;
  // a thread that cannot be created leaves its share to the others
  try {
    th.reserve(nt);
    for (int w = 1; w < nt; ++w)
      th.emplace_back([&, w] { err[w] = ring_worker(device, st, ring, w, to_host, host, dev, bytes, next); });
  } catch (...) {
  }
  err[0] = ring_worker(device, st, ring, 0, to_host, host, dev, bytes, next);
  for (auto& t : th) t.join();
  for (cudaError_t r : err)
    if (r != cudaSuccess) {
      cudaStreamSynchronize(st);  // nothing of a failed copy stays in flight
      return r;
    }
  return cudaSuccess;
}

// the ring, locked, if this copy goes through it (not when its slots cannot be
// allocated: the direct copy needs no pinned memory; nor on cudaStreamPerThread,
// which would be another stream in each of the copy's threads)
inline CopyRing* ring_for(int device, cudaStream_t st, bool to_host, const void* host, size_t bytes,
                          std::unique_lock<std::mutex>& lk) {
  CopyRing* r = ring_of(device);
  if (!r || st == cudaStreamPerThread || !ring_pays(to_host, host, bytes) || !host_pageable(host)) return nullptr;
  lk = std::unique_lock<std::mutex>(r->use, std::try_to_lock);
  if (!lk.owns_lock()) return nullptr;
  if (ensure_ring(*r) == cudaSuccess) return r;
  cudaGetLastError();
  return nullptr;
}

// device -> host, returns with the copy complete
inline cudaError_t copy_to_host(int device, cudaStream_t st, void* host, const void* dev, size_t bytes) {
  std::unique_lock<std::mutex> lk;
  if (CopyRing* r = ring_for(device, st, true, host, bytes, lk))
    return ring_copy(device, st, *r, true, static_cast<char*>(host), const_cast<char*>(static_cast<const char*>(dev)),
                     bytes);
  const cudaError_t e = cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, st);
  return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
}

// host -> device, in order with the stream's work (the host buffer may be
// reused once this returns)
inline cudaError_t copy_to_device(int device, cudaStream_t st, void* dev, const void* host, size_t bytes) {
  std::unique_lock<std::mutex> lk;
  if (CopyRing* r = ring_for(device, st, false, host, bytes, lk))
    return ring_copy(device, st, *r, false, const_cast<char*>(static_cast<const char*>(host)), static_cast<char*>(dev),
                     bytes);
  return cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, st);
}

}  // namespace iro
