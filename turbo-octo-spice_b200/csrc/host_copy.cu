// host_copy.cu — device-to-host copies of large results into pageable memory.
//
// The driver stages a pageable copy through its own pinned buffer on one
// thread, which for a result array that is new to the process also takes every
// page fault: 50 MB (the covariance of 2,500 bins) take 12 ms, here 4.5 to 5.  Up
// to four threads take 512 KB chunks in turn, each with two slots of a pinned
// buffer so that one chunk is on its way while the other is copied out.
// Below kStagedBytes starting the threads costs more than they save.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <string>
#include <thread>
#include <vector>

#include "engine_internal.h"

namespace tos {

namespace {
constexpr size_t kStagedBytes = 4u << 20;
constexpr int kSlotsPerThread = 2;
}  // namespace

bool HostStage::ready() {
  if (p) return true;
  for (int k = 0; k < kSlots; ++k)
    if (!ev[k] && cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming) != cudaSuccess) return false;
  void* q = nullptr;
  if (cudaMallocHost(&q, kSlots * kSlotBytes) != cudaSuccess) {
    cudaGetLastError();  // the plain copy takes over
    return false;
  }
  p = static_cast<unsigned char*>(q);
  return true;
}

void HostStage::release() {
  for (cudaEvent_t& v : ev) {
    if (v) cudaEventDestroy(v);
    v = nullptr;
  }
  if (p) cudaFreeHost(p);
  p = nullptr;
}

tos_status copy_out(tos_engine* e, void* dst, const void* src, size_t bytes) {
  cudaStream_t st = e->stream;
  cudaPointerAttributes at{};
  const bool pageable =
      cudaPointerGetAttributes(&at, dst) != cudaSuccess || at.type == cudaMemoryTypeUnregistered;
  cudaGetLastError();
  if (bytes < kStagedBytes || !pageable || !e->stage.ready()) {
    TOS_CUDA_TRY(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st));
    TOS_CUDA_TRY(cudaStreamSynchronize(st));
    return TOS_OK;
  }
  HostStage& S = e->stage;
  const size_t chunks = (bytes + HostStage::kSlotBytes - 1) / HostStage::kSlotBytes;
  std::atomic<size_t> next{0};
  std::atomic<int> err{(int)cudaSuccess};
  auto work = [&](int t) {
    cudaError_t r = cudaSetDevice(e->device);
    size_t at_slot[kSlotsPerThread];  // chunk in flight, or chunks
    auto issue = [&](int k) {
      const int slot = t * kSlotsPerThread + k;
      at_slot[k] = r == cudaSuccess ? std::min(next.fetch_add(1), chunks) : chunks;
      if (at_slot[k] == chunks) return;
      const size_t o = at_slot[k] * HostStage::kSlotBytes, n = std::min(HostStage::kSlotBytes, bytes - o);
      r = cudaMemcpyAsync(S.p + slot * HostStage::kSlotBytes, static_cast<const unsigned char*>(src) + o, n,
                          cudaMemcpyDeviceToHost, st);
      if (r == cudaSuccess) r = cudaEventRecord(S.ev[slot], st);
    };
    for (int k = 0; k < kSlotsPerThread; ++k) issue(k);
    for (int k = 0; at_slot[k] != chunks; k = (k + 1) % kSlotsPerThread) {
      const int slot = t * kSlotsPerThread + k;
      if (r == cudaSuccess) r = cudaEventSynchronize(S.ev[slot]);
      if (r == cudaSuccess) {
        const size_t o = at_slot[k] * HostStage::kSlotBytes, n = std::min(HostStage::kSlotBytes, bytes - o);
        std::memcpy(static_cast<unsigned char*>(dst) + o, S.p + slot * HostStage::kSlotBytes, n);
      }
      issue(k);
    }
    int ok = (int)cudaSuccess;
    if (r != cudaSuccess) err.compare_exchange_strong(ok, (int)r);
  };
  const int want = (int)std::min<size_t>(
      {(size_t)(HostStage::kSlots / kSlotsPerThread), std::max(1u, std::thread::hardware_concurrency()), chunks});
  std::vector<std::thread> others;
  try {
    others.reserve((size_t)want);
    for (int t = 1; t < want; ++t) others.emplace_back(work, t);
  } catch (...) {
    // fewer threads: those that run take the chunks
  }
  work(0);
  for (std::thread& t : others) t.join();
  if (err.load() != (int)cudaSuccess) {
    cudaStreamSynchronize(st);  // a chunk still on its way lands before its slot is used again
    return fail(TOS_ERR_CUDA, std::string("copy to the host: ") + cudaGetErrorString((cudaError_t)err.load()));
  }
  TOS_CUDA_TRY(cudaStreamSynchronize(st));
  return TOS_OK;
}

}  // namespace tos
