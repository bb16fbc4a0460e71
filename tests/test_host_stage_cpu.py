"""Staged host transfers (tg_stage.cuh) on the CPU: the header compiled against a stand-in for the
CUDA runtime whose copies are memcpy and whose calls fail on demand."""
import os
import subprocess

import pytest

from conftest import ROOT

RUNTIME = r"""
#pragma once
#include <atomic>
#include <cstddef>
#include <cstdlib>
#include <cstring>
typedef int cudaError_t;
typedef int* cudaEvent_t;
typedef void* cudaStream_t;
enum { cudaSuccess = 0, cudaErrorMemoryAllocation = 2, cudaErrorInvalidResourceHandle = 400 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice = 1, cudaMemcpyDeviceToHost = 2 };
enum { cudaMemoryTypeUnregistered = 0, cudaMemoryTypeHost = 1, cudaEventDisableTiming = 2 };
struct cudaPointerAttributes { int type; };
inline std::atomic<int> pinned_blocks{0}, events{0}, copies{0};
inline int fail_event = -1, fail_pinned = 0, made = 0;   // event creation that fails, pinned allocations that fail
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaSetDevice(int) { return cudaSuccess; }
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { a->type = 0; return cudaSuccess; }
inline cudaError_t cudaMallocHost(void** p, size_t n) {
  if (fail_pinned) return cudaErrorMemoryAllocation;
  *p = std::malloc(n);
  ++pinned_blocks;
  return cudaSuccess;
}
inline cudaError_t cudaFreeHost(void* p) { std::free(p); --pinned_blocks; return cudaSuccess; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  if (made++ == fail_event) return cudaErrorMemoryAllocation;
  *e = new int(0);
  ++events;
  return cudaSuccess;
}
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; --events; return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
  return e ? cudaSuccess : cudaErrorInvalidResourceHandle;
}
inline cudaError_t cudaEventSynchronize(cudaEvent_t e) { return e ? cudaSuccess : cudaErrorInvalidResourceHandle; }
inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(d, s, n);
  ++copies;
  return cudaSuccess;
}
"""

MAIN = r"""
#include <cstdio>
#include <vector>
#include "tg_stage.cuh"
int main(int argc, char** argv) {
  fail_event = std::atoi(argv[1]);
  fail_pinned = std::atoi(argv[2]);
  tg::HostStage st;
  const size_t least = tg::kStageLeast, pays = tg::kStagePays, piece = tg::kStagePiece;
  for (int round = 0; round < 2; ++round) {
    for (size_t n : {least - 1, least, 9 * piece + 5, pays + 1}) {
      for (bool up : {true, false}) {
        std::vector<unsigned char> a(n), b(n, 0);
        for (size_t i = 0; i < n; ++i) a[i] = (unsigned char)(i * 131 + i / 251 + round);
        copies = 0;
        if (st.copy(0, nullptr, b.data(), a.data(), n, up) != cudaSuccess) return 1;
        if (a != b) return 2;
        const int want = st.pinned && n >= least ? (int)((n + piece - 1) / piece) : 1;
        if (copies != want) return 3;
        if (events != (st.pinned ? 2 * tg::kStageThreads : 0) || pinned_blocks != (st.pinned ? 1 : 0)) return 4;
      }
    }
  }
  if ((st.pinned != nullptr) != (fail_pinned == 0)) return 5;   // a failed event is tried again later
  st.release();
  return events == 0 && pinned_blocks == 0 ? 0 : 6;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("stage")
    (d / "cuda_runtime.h").write_text(RUNTIME)
    (d / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-I", str(d), "-I",
                    os.path.join(ROOT, "titan_b200", "csrc"), str(d / "main.cpp"), "-o", str(d / "stage")], check=True)
    return str(d / "stage")


@pytest.mark.parametrize("event,pinned", [(-1, 0), (0, 0), (5, 0), (15, 0), (-1, 1)])
def test_copies_with_and_without_staging(program, event, pinned):
    """Every copy arrives whole; an event or a pinned buffer that cannot be made leaves the plain
    copies, with nothing half made, and is tried again by a later one."""
    assert subprocess.run([program, str(event), str(pinned)], timeout=60).returncode == 0
