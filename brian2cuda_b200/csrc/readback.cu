// Large device-to-host reads: state variables and synaptic variables into the caller's array.
//
// A copy into pageable memory goes through the driver's staging in one thread, and a fresh
// array's pages are faulted in by that thread as they are written: 4 GB/s for the weights of 1e7
// synapses.  Here the value moves in chunks of 1 MB through page-locked slots,
// several host threads each with a slot of its own: while one thread's chunk crosses the bus the
// others write theirs into the caller's pages.  A value that has to be gathered on the device
// first (a synapse variable in input order) is gathered chunk by chunk into the slot's device
// half, so no buffer of the value's size is allocated.  The copies run on the net's stream, in
// any order; the caller's array is complete on return.  Without memory for the slots the plain
// copy runs.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <new>
#include <system_error>
#include <thread>
#include <vector>

#include "b2b_internal.h"

namespace b2b {

namespace {

constexpr size_t kReadChunk = (size_t)1 << 20;
constexpr int kReadSlots = 6;
// A plain array below this is one copy: us for 0.6e6 / 0.8e6 / 1e6 / 2e6 floats, copied / by slots, into
// pages in use 160 / 176, 200 / 260, 235 / 235, 430 / 440, into new ones (1e6, 2e6) 1830 / 680, 2100 / 970.
// (A gathered value is spared its buffer as well: 0.6e6 855 / 333.)
constexpr size_t kReadArrayMin = 4000000;

// Sets of slots not in use.  Page-locking a set takes milliseconds, so a set outlives the read
// (and the net) that needed it, at most kKeptSets of them, until the last net is destroyed.  A read
// takes a set of its device out of the pool for its duration, so nets of several threads never
// share one.
struct ReadSlots {
  int device = 0;
  void* pinned = nullptr;
  void* dev = nullptr;
  cudaEvent_t ev[kReadSlots] = {};
};
constexpr int kKeptSets = 2;
std::mutex g_mutex;
ReadSlots g_free[kKeptSets];
int g_n_free = 0, g_nets = 0;

void release(ReadSlots& S) {
  cudaSetDevice(S.device);
  if (S.pinned) cudaFreeHost(S.pinned);
  if (S.dev) cudaFree(S.dev);
  for (cudaEvent_t e : S.ev)
    if (e) cudaEventDestroy(e);
}

bool take(int device, ReadSlots* out) {
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    for (int i = 0; i < g_n_free; ++i)
      if (g_free[i].device == device) {
        *out = g_free[i];
        g_free[i] = g_free[--g_n_free];
        return true;
      }
  }
  ReadSlots S;
  S.device = device;
  bool ok = cudaMallocHost(&S.pinned, kReadSlots * kReadChunk) == cudaSuccess &&
            cudaMalloc(&S.dev, kReadSlots * kReadChunk) == cudaSuccess;
  for (int t = 0; t < kReadSlots && ok; ++t)
    ok = cudaEventCreateWithFlags(&S.ev[t], cudaEventDisableTiming) == cudaSuccess;
  if (!ok) {
    cudaGetLastError();
    release(S);
    return false;
  }
  *out = S;
  return true;
}

// After a read whose copies have completed.
void give_back(ReadSlots& S) {
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    if (g_n_free < kKeptSets && g_nets > 0) {
      g_free[g_n_free++] = S;
      return;
    }
  }
  release(S);
}

}  // namespace

void readback_net_created() {
  std::lock_guard<std::mutex> lock(g_mutex);
  ++g_nets;
}

void readback_net_destroyed() {
  std::lock_guard<std::mutex> lock(g_mutex);
  if (--g_nets > 0) return;
  int device = 0;                      // the caller's, which the sets' need not be
  const bool known = cudaGetDevice(&device) == cudaSuccess;
  while (g_n_free > 0) release(g_free[--g_n_free]);
  if (known) cudaSetDevice(device);
}

bool read_back_worth(size_t bytes) { return bytes >= 2 * kReadChunk; }

cudaError_t read_back(b2b_net* net, void* host, size_t bytes, const ReadSource& source) {
  ReadSlots S;
  if (!take(net->cfg.device, &S)) return cudaErrorMemoryAllocation;
  const size_t chunks = (bytes + kReadChunk - 1) / kReadChunk;
  std::atomic<size_t> next{0};
  std::atomic<int> error{cudaSuccess};
  auto work = [&](int t) {
    uint8_t* pin = static_cast<uint8_t*>(S.pinned) + (size_t)t * kReadChunk;
    uint8_t* dev = static_cast<uint8_t*>(S.dev) + (size_t)t * kReadChunk;
    cudaError_t e = cudaSetDevice(net->cfg.device);
    for (size_t c = next++; c < chunks && e == cudaSuccess && error == cudaSuccess; c = next++) {
      const size_t off = c * kReadChunk, len = std::min(kReadChunk, bytes - off);
      const void* src = nullptr;
      e = source(off, len, dev, &src, net->stream);
      if (e == cudaSuccess) e = cudaMemcpyAsync(pin, src, len, cudaMemcpyDeviceToHost, net->stream);
      if (e == cudaSuccess) e = cudaEventRecord(S.ev[t], net->stream);
      if (e == cudaSuccess) e = cudaEventSynchronize(S.ev[t]);
      if (e == cudaSuccess) memcpy(static_cast<uint8_t*>(host) + off, pin, len);
    }
    if (e != cudaSuccess) error = e;
  };
  std::vector<std::thread> helpers;
  const unsigned cores = std::thread::hardware_concurrency();
  const size_t threads = std::min<size_t>({(size_t)kReadSlots, chunks, cores ? cores : 1});
  try {
    helpers.reserve(threads);
    for (size_t t = 1; t < threads; ++t) helpers.emplace_back(work, (int)t);
  } catch (const std::system_error&) {
    // fewer threads share the chunks
  } catch (const std::bad_alloc&) {
  }
  work(0);
  for (std::thread& h : helpers) h.join();
  // after an error a copy into a slot may still be under way
  if (error != cudaSuccess) cudaStreamSynchronize(net->stream);
  give_back(S);
  return (cudaError_t)error.load();
}

cudaError_t read_array(b2b_net* net, void* host, const void* dev, size_t bytes) {
  if (bytes >= kReadArrayMin) {
    try {
      const cudaError_t e = read_back(
          net, host, bytes,
          [dev](size_t off, size_t, void*, const void** src, cudaStream_t) {
            *src = static_cast<const uint8_t*>(dev) + off;
            return cudaSuccess;
          });
      if (e != cudaErrorMemoryAllocation) return e;
    } catch (const std::bad_alloc&) {
    }
  }
  const cudaError_t e = cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, net->stream);
  return e != cudaSuccess ? e : cudaStreamSynchronize(net->stream);
}

}  // namespace b2b
