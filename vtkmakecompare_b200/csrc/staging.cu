// staging.cu -- copies between a caller's pageable arrays and the GPU through
// pinned slots.
//
// The Fortran drop-ins get ordinary host memory.  A driver copy from or to it
// runs on one thread, and a box of a padded field row by row: MKP on
// 96x64x96 spent 25 of its 27 ms in 18 such copies (86 MB); the call now takes
// 3.6 ms.  Here several threads move the data between the arrays and a fixed
// set of pinned slots while the DMA engine empties and fills the others; a box
// comes over as whole rows and only its entries are written to the caller's
// array.
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <thread>
#include <vector>

#include "common.cuh"

namespace nse {

namespace {

constexpr int kThreads = 8, kSlots = 2;   // slots of each thread
constexpr size_t kSlot = 512 * 1024;      // bytes of a slot: 8 MB pinned in all
constexpr size_t kMin = 1024 * 1024;      // smaller transfers are not split

// The slots, kept between calls (pinning them takes longer than a call) and
// freed at exit.  One set of copies uses them at a time.
struct Pool {
  std::mutex mu;
  char* base = nullptr;
  cudaEvent_t ev[kThreads * kSlots] = {};
  bool ready() {
    if (base) return true;
    if (cudaHostAlloc((void**)&base, kThreads * kSlots * kSlot, cudaHostAllocPortable) != cudaSuccess) {
      cudaGetLastError();
      base = nullptr;
      return false;
    }
    for (auto& e : ev)
      if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
        cudaGetLastError();
        release();
        return false;
      }
    static bool registered = false;
    if (!registered) registered = atexit([]() { pool().release(); }) == 0;
    return true;
  }
  void release() {
    for (auto& e : ev) {
      if (e) cudaEventDestroy(e);
      e = nullptr;
    }
    if (base) cudaFreeHost(base);
    base = nullptr;
  }
  static Pool& pool() {
    static Pool* p = new Pool;  // (never destroyed: the exit handler frees what it holds)
    return *p;
  }
};

struct Chunk {
  const HostCopy* c;
  size_t b0, b1;  // bytes of the copied region
};

void scatter(const Chunk& k, const char* slot) {
  const HostCopy& c = *k.c;
  char* host = static_cast<char*>(c.host);
  if (c.per == 1 && c.width == c.pitch) {
    memcpy(host + k.b0, slot, k.b1 - k.b0);
    return;
  }
  for (size_t b = k.b0; b < k.b1; b += c.pitch) {
    const int r = (int)((b / c.pitch) % c.per);
    if (r >= c.lo && r <= c.hi) memcpy(host + b + c.off, slot + (b - k.b0) + c.off, c.width);
  }
}

// thread t's chunks t, t + nt, ... through its own slots
bool run_chunks(const std::vector<Chunk>& ch, int t, int nt, bool to_device, Pool& P, int dev,
                cudaStream_t s) {
  if (cudaSetDevice(dev) != cudaSuccess) return false;
  bool ok = true;
  const int n = t < (int)ch.size() ? ((int)ch.size() - t + nt - 1) / nt : 0;
  auto slot = [&](int q) { return P.base + (size_t)(t * kSlots + q % kSlots) * kSlot; };
  auto ev = [&](int q) { return P.ev[t * kSlots + q % kSlots]; };
  auto chunk = [&](int q) -> const Chunk& { return ch[t + (size_t)q * nt]; };
  auto dma = [&](int q) {
    const Chunk& k = chunk(q);
    char* d = static_cast<char*>(k.c->dev) + k.b0;
    ok = ok && cudaMemcpyAsync(to_device ? d : slot(q), to_device ? slot(q) : d, k.b1 - k.b0,
                               to_device ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost,
                               s) == cudaSuccess;
    ok = ok && cudaEventRecord(ev(q), s) == cudaSuccess;
  };
  if (to_device) {
    for (int q = 0; ok && q < n; ++q) {
      if (q >= kSlots) ok = cudaEventSynchronize(ev(q)) == cudaSuccess;
      if (!ok) break;
      memcpy(slot(q), static_cast<const char*>(chunk(q).c->host) + chunk(q).b0,
             chunk(q).b1 - chunk(q).b0);
      dma(q);
    }
    // the slots may be refilled by the next set of copies: wait for the DMA
    for (int q = std::max(0, n - kSlots); q < n; ++q) ok = cudaEventSynchronize(ev(q)) == cudaSuccess && ok;
    return ok;
  }
  for (int q = 0; q < std::min(n, kSlots); ++q) dma(q);
  for (int q = 0; ok && q < n; ++q) {
    ok = cudaEventSynchronize(ev(q)) == cudaSuccess;
    if (!ok) break;
    scatter(chunk(q), slot(q));
    if (q + kSlots < n) dma(q + kSlots);
  }
  return ok;
}

// one copy as the driver does it
bool plain(const HostCopy& c, bool to_device, cudaStream_t s) {
  if (to_device)
    return cudaMemcpyAsync(c.dev, c.host, c.bytes, cudaMemcpyHostToDevice, s) == cudaSuccess;
  if (c.per == 1 && c.width == c.pitch)
    return cudaMemcpyAsync(c.host, c.dev, c.bytes, cudaMemcpyDeviceToHost, s) == cudaSuccess;
  cudaMemcpy3DParms p;
  memset(&p, 0, sizeof(p));
  p.srcPtr = make_cudaPitchedPtr(c.dev, c.pitch, c.pitch, c.per);
  p.dstPtr = make_cudaPitchedPtr(c.host, c.pitch, c.pitch, c.per);
  p.srcPos = make_cudaPos(c.off, c.lo, 0);
  p.dstPos = p.srcPos;
  p.extent = make_cudaExtent(c.width, c.hi - c.lo + 1, c.bytes / (c.pitch * c.per));
  p.kind = cudaMemcpyDeviceToHost;
  return cudaMemcpy3DAsync(&p, s) == cudaSuccess;
}

}  // namespace

bool host_copies(const HostCopy* list, int n, bool to_device, cudaStream_t s) {
  size_t total = 0;
  bool fits = true;  // rows of a box stay whole in a slot
  for (int q = 0; q < n; ++q) {
    total += list[q].bytes;
    fits = fits && (list[q].per == 1 || list[q].pitch <= kSlot);
  }
  Pool& P = Pool::pool();
  std::unique_lock<std::mutex> lk(P.mu, std::defer_lock);
  bool ok = true;
  if (total >= kMin && fits && lk.try_lock() && P.ready()) {
    int dev = 0;
    cudaGetDevice(&dev);
    std::vector<Chunk> ch;
    for (int q = 0; q < n; ++q) {
      const HostCopy& c = list[q];
      const size_t step = c.pitch >= kSlot ? kSlot : kSlot / c.pitch * c.pitch;
      for (size_t b = 0; b < c.bytes; b += step) ch.push_back({&c, b, std::min(c.bytes, b + step)});
    }
    const int nt = std::max(1, std::min({kThreads, (int)std::thread::hardware_concurrency(),
                                         (int)ch.size()}));
    std::atomic<bool> good{true};
    std::vector<std::thread> th;
    int started = 1;
    try {
      for (; started < nt; ++started) {
        const int t = started;
        th.emplace_back([&, t]() {
          if (!run_chunks(ch, t, nt, to_device, P, dev, s)) good = false;
        });
      }
    } catch (...) {  // no thread to be had: this one does the rest
    }
    if (!run_chunks(ch, 0, nt, to_device, P, dev, s)) good = false;
    for (int t = started; t < nt; ++t)
      if (!run_chunks(ch, t, nt, to_device, P, dev, s)) good = false;
    for (auto& t : th) t.join();
    ok = good;
  } else {
    for (int q = 0; ok && q < n; ++q) ok = plain(list[q], to_device, s);
    // (a page-locked array's copy is still under way here)
    if (ok && !to_device) ok = cudaStreamSynchronize(s) == cudaSuccess;
  }
  if (ok) return true;
  const cudaError_t e = cudaGetLastError();
  // copies that were queued before one failed still use the slots and the caller's
  // arrays: wait for them while the slots are this call's
  cudaStreamSynchronize(s);
  return cuda_ok(e != cudaSuccess ? e : cudaErrorUnknown, "copy between a host array and the GPU");
}

}  // namespace nse
