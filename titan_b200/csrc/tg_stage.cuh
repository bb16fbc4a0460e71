// Large transfers between pageable host arrays and the device.
//
// cudaMemcpyAsync stages those through one thread of the driver (and on a fresh result array that
// thread takes every page fault); here up to kStageThreads threads of this call each move their
// part in pieces of kStagePiece through two pinned buffers of the context, copying one piece while
// the other is on the link.  Transfers below kStageLeast (a few pieces, the least that several
// threads can share), and arrays that are pinned already, go to cudaMemcpyAsync.  When it was
// brought in, a call with a result of 41 MB went from 108 to 101 ms, one with four results of
// 6.7 MB from 215 to 211 ms.  Pinning the buffers takes about 10 ms, what they save on 64 MB
// (kStagePays): a context makes them when it has been asked to move that much.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstring>
#include <thread>
#include <vector>

namespace tg {

constexpr int kStageThreads = 8;
constexpr size_t kStagePiece = (size_t)1 << 20;
constexpr size_t kStageLeast = (size_t)4 << 20;
constexpr size_t kStagePays = (size_t)64 << 20;

struct HostStage {
  char* pinned = nullptr;   // two pieces per thread
  cudaEvent_t events[2 * kStageThreads] = {};
  size_t moved = 0;         // bytes of large pageable transfers so far

  void release() {
    for (cudaEvent_t& e : events) {
      if (e) cudaEventDestroy(e);
      e = nullptr;
    }
    if (pinned) cudaFreeHost(pinned);
    pinned = nullptr;
  }

  // the buffers and an event for each, or (false) nothing
  bool make() {
    void* p = nullptr;
    if (cudaMallocHost(&p, 2 * kStageThreads * kStagePiece) == cudaSuccess) {
      pinned = static_cast<char*>(p);
      bool ok = true;
      for (cudaEvent_t& e : events) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
      if (ok) return true;
      release();
    }
    cudaGetLastError();
    return false;
  }

  // The source of an upload may be reused, and the destination of a download read, on return.
  cudaError_t copy(int device, cudaStream_t stream, void* dst, const void* src, size_t bytes, bool to_device) {
    const cudaMemcpyKind kind = to_device ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost;
    auto plain = [&]() {
      const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, kind, stream);
      return e != cudaSuccess ? e : cudaStreamSynchronize(stream);
    };
    if (bytes < kStageLeast) return plain();
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, to_device ? src : dst) != cudaSuccess) cudaGetLastError();
    else if (at.type != cudaMemoryTypeUnregistered) return plain();
    moved += bytes;
    if (!pinned && (moved < kStagePays || !make())) return plain();
    const size_t pieces = (bytes + kStagePiece - 1) / kStagePiece;
    const int nt = (int)std::min<size_t>(std::min<size_t>(kStageThreads, pieces),
                                         std::max(1u, std::thread::hardware_concurrency()));
    std::atomic<int> err{(int)cudaSuccess};
    auto work = [&](int t) {   // pieces t, t + nt, ..
      auto fail = [&](cudaError_t e) {
        if (e == cudaSuccess) return false;
        err.store((int)e);
        return true;
      };
      if (fail(cudaSetDevice(device))) return;
      char* buf[2] = {pinned + (size_t)(2 * t) * kStagePiece, pinned + (size_t)(2 * t + 1) * kStagePiece};
      cudaEvent_t* ev = events + 2 * t;
      auto part = [&](size_t i) { return std::min(kStagePiece, bytes - i * kStagePiece); };
      size_t turn = 0;
      if (to_device) {
        for (size_t i = t; i < pieces; i += nt, ++turn) {
          const int b = (int)(turn & 1);
          if (turn >= 2 && fail(cudaEventSynchronize(ev[b]))) return;
          std::memcpy(buf[b], static_cast<const char*>(src) + i * kStagePiece, part(i));
          if (fail(cudaMemcpyAsync(static_cast<char*>(dst) + i * kStagePiece, buf[b], part(i), kind, stream))) return;
          if (fail(cudaEventRecord(ev[b], stream))) return;
        }
        for (int b = 0; b < 2 && b < (int)turn; ++b)
          if (fail(cudaEventSynchronize(ev[b]))) return;
      } else {
        auto fetch = [&](size_t i, int b) {
          return fail(cudaMemcpyAsync(buf[b], static_cast<const char*>(src) + i * kStagePiece, part(i), kind, stream)) ||
                 fail(cudaEventRecord(ev[b], stream));
        };
        if (fetch(t, 0)) return;
        for (size_t i = t; i < pieces; i += nt, ++turn) {
          const int b = (int)(turn & 1);
          if (i + nt < pieces && fetch(i + nt, b ^ 1)) return;
          if (fail(cudaEventSynchronize(ev[b]))) return;
          std::memcpy(static_cast<char*>(dst) + i * kStagePiece, buf[b], part(i));
        }
      }
    };
    std::vector<std::thread> threads;
    int started = 0;
    try {
      threads.reserve(nt);
      for (int t = 1; t < nt; ++t) {
        threads.emplace_back(work, t);
        ++started;
      }
    } catch (...) {   // no more threads to be had: their parts are done here
    }
    work(0);
    for (int t = started + 1; t < nt; ++t) work(t);
    for (auto& th : threads) th.join();
    if (err.load() != (int)cudaSuccess) cudaStreamSynchronize(stream);   // no copy still reads the buffers
    return (cudaError_t)err.load();
  }
};

}  // namespace tg
