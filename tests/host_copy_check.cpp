// csrc/host_copy.h against a CUDA runtime of this file's own: device memory is
// host memory, and a stream runs its queued operations only when an event
// recorded in it, or the stream, is waited for: the latest moment that the
// CUDA ordering rules allow.  argv[1] names the check; exits 0 when it holds.
#include "host_copy.h"

#include <cstdio>
#include <cstdlib>
#include <deque>
#include <map>
#include <string>

namespace {

struct Op {
  void* dst;
  const void* src;
  size_t bytes;
};
struct Stream {
  std::deque<Op> queue;
  size_t done = 0, queued = 0;
};
struct Event {
  Stream* st = nullptr;
  size_t at = 0;
};
std::mutex g_mutex;
std::map<cudaStream_t, Stream> g_streams;
bool g_fail_pinned = false;
int g_pinned_live = 0, g_copies = 0;

// every thread has its own cudaStreamPerThread
Stream& stream_of(cudaStream_t st) {
  static thread_local char mine;
  return g_streams[st == cudaStreamPerThread ? reinterpret_cast<cudaStream_t>(&mine) : st];
}

void run_until(Stream& s, size_t at) {
  while (s.done < at) {
    std::memcpy(s.queue.front().dst, s.queue.front().src, s.queue.front().bytes);
    s.queue.pop_front();
    ++s.done;
  }
}

}  // namespace

extern "C" {
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
  a->type = cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned) {
  if (g_fail_pinned) return cudaErrorMemoryAllocation;
  *p = std::malloc(bytes);
  ++g_pinned_live;
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  std::free(p);
  --g_pinned_live;
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = reinterpret_cast<cudaEvent_t>(new Event);
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  delete reinterpret_cast<Event*>(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) {
  std::lock_guard<std::mutex> lk(g_mutex);
  Stream& s = stream_of(st);
  *reinterpret_cast<Event*>(e) = Event{&s, s.queued};
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  std::lock_guard<std::mutex> lk(g_mutex);
  const Event& v = *reinterpret_cast<Event*>(e);
  if (v.st) run_until(*v.st, v.at);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t bytes, cudaMemcpyKind, cudaStream_t st) {
  std::lock_guard<std::mutex> lk(g_mutex);
  Stream& s = stream_of(st);
  s.queue.push_back(Op{dst, src, bytes});
  ++s.queued;
  ++g_copies;
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st) {
  std::lock_guard<std::mutex> lk(g_mutex);
  Stream& s = stream_of(st);
  run_until(s, s.queued);
  return cudaSuccess;
}
}

using namespace iro;
using Bytes = std::vector<unsigned char>;

static cudaStream_t stream(long k) { return reinterpret_cast<cudaStream_t>(0x1000 * k); }
static Bytes pattern(size_t n, unsigned seed) {
  Bytes b(n);
  for (size_t i = 0; i < n; ++i) b[i] = static_cast<unsigned char>((i >> 8) * 37 + i + seed);
  return b;
}
static int verdict(bool ok, const char* what) {
  if (!ok) std::printf("%s\n", what);
  return ok ? 0 : 1;
}

// An upload on one context's stream, then a download on another's: the second
// copy's DMAs must not touch a slot before the first's have read it.
static int other_context(size_t up, size_t down) {
  const Bytes a = pattern(up, 1), b = pattern(down, 2);
  Bytes dev_a(up), dev_b = b, host_b(down);
  ring_attach(0);
  ring_attach(0);
  copy_to_device(0, stream(1), dev_a.data(), a.data(), up);
  copy_to_host(0, stream(2), host_b.data(), dev_b.data(), down);
  cudaStreamSynchronize(stream(1));
  int rc = verdict(dev_a == a, "the upload was overwritten") + verdict(host_b == b, "wrong download");
  // as two contexts are destroyed: the slots go with the last one
  copy_to_device(0, stream(2), dev_b.data(), b.data(), down);
  copy_to_device(0, stream(1), dev_a.data(), a.data(), up);
  cudaStreamSynchronize(stream(1));
  ring_detach(0);
  cudaStreamSynchronize(stream(2));
  ring_detach(0);
  return rc + verdict(g_pinned_live == 0, "pinned slots kept") + verdict(dev_a == a && dev_b == b, "wrong uploads");
}

// What a copy queues: one operation when it is direct, one per MiB through the slots
static int copies(bool up, void* host, size_t n) {
  static Bytes dev(size_t(80) << 20);
  const int before = g_copies;
  if (up) copy_to_device(0, stream(1), dev.data(), host, n);
  else copy_to_host(0, stream(1), host, dev.data(), n);
  cudaStreamSynchronize(stream(1));
  return g_copies - before;
}

// Which copies go through the slots: by direction, size and whether the
// destination was touched before
static int route() {
  const size_t MB = size_t(1) << 20;
  Bytes touched(80 * MB, 1);
  int rc = 0;
  ring_attach(0);
  auto expect = [&](bool up, void* host, size_t n, bool slots, const char* what) {
    const int k = copies(up, host, n), want = slots ? int((n + MB - 1) / MB) : 1;
    if (k != want) std::printf("%zu bytes: %d operations instead of %d, ", n, k, want);
    rc += verdict(k == want, what);
  };
  for (size_t n : {MB, 4 * MB, 8 * MB, 10 * MB - 8}) expect(true, touched.data(), n, false, "upload");
  for (size_t n : {10 * MB, 17 * MB + 8, 64 * MB}) expect(true, touched.data(), n, true, "upload");
  for (size_t n : {MB, 4 * MB, 16 * MB, 32 * MB - 8}) expect(false, touched.data(), n, false, "touched download");
  for (size_t n : {32 * MB, 40 * MB + 8, 80 * MB}) expect(false, touched.data(), n, true, "touched download");
  for (size_t n : {4 * MB - 8, 4 * MB, 8 * MB + 8, 24 * MB}) {
    // any alignment, and memory that ends with the destination
    const size_t room = (n + 8191) / 4096 * 4096;
    char* p = static_cast<char*>(mmap(nullptr, room, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
    expect(false, p + (room - n), n, n >= 4 * MB, "untouched download");
    expect(false, p + (room - n), n, n >= 32 * MB, "the same again, touched now");
    munmap(p, room);
  }
  ring_detach(0);
  return rc;
}

// The slots cannot be had: copies of every size take the direct path, and the
// slots again once they can
static int no_pinned_memory() {
  const size_t n = (size_t(40) << 20) + 8;
  const Bytes a = pattern(n, 3);
  Bytes dev(n), back(n);
  int rc = 0;
  ring_attach(0);
  for (bool fail : {true, false, true}) {
    g_fail_pinned = fail;
    std::fill(dev.begin(), dev.end(), 0);
    std::fill(back.begin(), back.end(), 0);
    rc += verdict(copy_to_device(0, stream(1), dev.data(), a.data(), n) == cudaSuccess, "upload refused");
    rc += verdict(copy_to_host(0, stream(1), back.data(), dev.data(), n) == cudaSuccess, "download refused");
    rc += verdict(dev == a && back == a, "wrong bytes");
  }
  ring_detach(0);
  return rc + verdict(g_pinned_live == 0, "pinned slots kept");
}

// A context on cudaStreamPerThread, a handle that means another stream in each
// thread: copies stay in order with the calling thread's work
static int per_thread_stream() {
  const size_t n = size_t(40) << 20;
  const Bytes a = pattern(n, 4), b = pattern(n, 5);
  Bytes dev(n), other(n), back(n);
  ring_attach(0);
  cudaMemcpyAsync(dev.data(), a.data(), n, cudaMemcpyDeviceToDevice, cudaStreamPerThread);
  copy_to_host(0, cudaStreamPerThread, back.data(), dev.data(), n);
  int rc = verdict(back == a, "the download overtook the work before it");
  cudaMemcpyAsync(other.data(), dev.data(), n, cudaMemcpyDeviceToDevice, cudaStreamPerThread);
  copy_to_device(0, cudaStreamPerThread, dev.data(), b.data(), n);
  cudaStreamSynchronize(cudaStreamPerThread);
  rc += verdict(other == a && dev == b, "the upload overtook the work before it");
  ring_detach(0);
  return rc;
}

int main(int argc, char** argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  const size_t MB = size_t(1) << 20;
  if (what == "other_context") {
    int rc = 0;
    for (size_t up : {10 * MB, 16 * MB, 40 * MB + 24})
      for (size_t down : {32 * MB, 33 * MB + 8, 64 * MB}) rc += other_context(up, down);
    return rc;
  }
  if (what == "route") return route();
  if (what == "per_thread_stream") return per_thread_stream();
  if (what == "no_pinned_memory") return no_pinned_memory();
  std::printf("unknown check\n");
  return 2;
}
