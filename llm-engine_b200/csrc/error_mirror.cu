// Host-visible record of bounded waits that ran out.
//
// Every wait inside the kernels is bounded; a wait that runs out leaves a bit in a device word
// (pkv_debug_device_flags reads it, synchronising) and, so that the caller learns of it without
// synchronising, in one pinned host word that the kernels can store to.  The attention entry points
// look at that word before they enqueue anything, and so do the block copies for a copy's bit: the call
// that follows an incomplete launch returns PKV_E_CUDA once (the word is cleared by the report), in the
// manner of CUDA's own asynchronous errors.  The launch after that runs normally: nothing is disabled.
#include <cuda_runtime.h>

#include <cstring>
#include <mutex>

#include "status.hpp"

namespace pkv {
namespace {
std::mutex g_mu;
unsigned int* g_mirror = nullptr;   // cudaHostAlloc'd (portable, mapped): kWords words, valid on every device
constexpr int kWords = 2;           // the attention kernels' and the block copies': they store their bit, they do not add it
bool g_tried = false;
unsigned int g_plain = 0;           // what pkv_debug_set_reported_flags recorded (works without a device)
}  // namespace

// The pinned words, created on first use when `create` is set.  The one allocating call this makes
// (cudaHostAlloc of 64 bytes, once per process) is kept away from callers that must not allocate:
// they pass create = false and get the words only if somebody else made them already.
unsigned int* error_mirror(bool create) {
  std::lock_guard<std::mutex> lock(g_mu);
  if (g_mirror || !create || g_tried) return g_mirror;
  g_tried = true;
  void* p = nullptr;
  // the first call may be one that is being captured into a graph, which an allocation must not end
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  cudaThreadExchangeStreamCaptureMode(&mode);
  const cudaError_t e = cudaHostAlloc(&p, 64, cudaHostAllocPortable | cudaHostAllocMapped);
  cudaThreadExchangeStreamCaptureMode(&mode);
  if (e == cudaSuccess && p) {
    std::memset(p, 0, 64);
    __atomic_store_n(&g_mirror, static_cast<unsigned int*>(p), __ATOMIC_RELEASE);
  } else {
    cudaGetLastError();
  }
  return g_mirror;
}

// Takes those of `bits` that are recorded.
unsigned int take_error_mirror(unsigned int bits) {
  // the common case -- nothing recorded -- is three plain loads, no lock and no write
  unsigned int* m = __atomic_load_n(&g_mirror, __ATOMIC_ACQUIRE);
  unsigned int seen = __atomic_load_n(&g_plain, __ATOMIC_RELAXED);
  for (int i = 0; m && i < kWords; ++i) seen |= __atomic_load_n(m + i, __ATOMIC_RELAXED);
  if ((seen & bits) == 0) return 0;
  std::lock_guard<std::mutex> lock(g_mu);
  unsigned int v = g_plain & bits;
  g_plain &= ~bits;
  for (int i = 0; g_mirror && i < kWords; ++i) v |= __atomic_fetch_and(g_mirror + i, ~bits, __ATOMIC_ACQ_REL) & bits;
  return v;
}

int check_error_mirror(const char* fn, unsigned int bits) {
  const unsigned int v = take_error_mirror(bits);
  if (!v) return PKV_OK;
  return fail(PKV_E_CUDA,
              "%s: an earlier launch gave up on a bounded wait (flags 0x%x: 1 TMA producer, 2 tile consumer, 4 prefill "
              "pipeline, 8 peer GPU, 16 block copy) and left its output incomplete; this call enqueued nothing, the next one runs normally",
              fn, v);
}

}  // namespace pkv

extern "C" int pkv_debug_set_reported_flags(unsigned int flags) {
  std::lock_guard<std::mutex> lock(pkv::g_mu);
  pkv::g_plain |= flags;
  return PKV_OK;
}
