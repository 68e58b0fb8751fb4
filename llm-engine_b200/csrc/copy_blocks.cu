// Prefix-cache copy-on-write block copy (include/pkv.h, "block copy").
//
// A block of one pool is block_size * kv_dim elements of contiguous memory, so the
// copy of pair (src, dst) in pool p is a straight memcpy of block_bytes.  Bit-exact by
// construction.
#include <algorithm>

#include "common.cuh"
#include "launch_util.hpp"
#include "status.hpp"
#include "tma_util.hpp"

namespace pkv {
unsigned int* error_mirror(bool create);                 // error_mirror.cu
int check_error_mirror(const char* fn, unsigned int bits);

__device__ unsigned int g_pkv_copy_error = 0;

namespace {

constexpr unsigned kErrCopyWait = 16u;   // bit of the device error word: a block's bytes did not arrive in time

__device__ __forceinline__ void copy_give_up(unsigned int* host_err) {
  atomicOr(&g_pkv_copy_error, kErrCopyWait);
  if (host_err) {
    *reinterpret_cast<volatile unsigned int*>(host_err) = kErrCopyWait;
    __threadfence_system();
  }
}

constexpr int kCopyThreads = 128;

struct TwoPools { void* p[2]; };

// The copies are dealt over persistent blocks of one warp whose first lane streams them through a ring in
// shared memory with bulk copies (global -> shared -> global, up to 8 KB each), so that an SM keeps up to
// 190 KB of reads and writes in flight.  HBM-bound: 127 pairs x 44 pools of 8 KB (91.6 MB moved) 18.6 us with a
// thread block of ordinary 16-byte loads and stores per (pair, pool), 16.8 us (5.4 TB/s) this way; smaller waves
// gain as much (32 pairs, within L2: 6.0 -> 4.9 us).  Two to six blocks per SM measured alike.
constexpr int kBulkBytes = 8192, kBulkStages = 4, kBulkBlocksPerSm = 6;

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst), "l"(src),
               "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void bulk_store(void* dst, uint32_t src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
}

template <bool FROM_ARRAY>
__global__ void __launch_bounds__(32) copy_blocks_bulk_kernel(TwoPools two, void* const* __restrict__ pools,
                                                              const int* __restrict__ pairs, unsigned n_pairs, unsigned long long block_bytes,
                                                              unsigned long long pieces, unsigned long long n_tasks,
                                                              unsigned int* host_err) {
  extern __shared__ __align__(128) unsigned char ring[];
  __shared__ __align__(8) unsigned long long full[kBulkStages];
  const int lane = threadIdx.x;
  if (lane == 0) {
    for (int i = 0; i < kBulkStages; ++i) mbar_init(smem_u32(&full[i]), 1);
    mbar_fence_init();
  }
  __syncwarp();
  pdl_wait();
  // Copy t: piece t % pieces of pair (t / pieces) % n_pairs in pool t / pieces / n_pairs; this block's are
  // blockIdx.x, blockIdx.x + gridDim.x, ...  Lanes look up 32 of them at a time; lane 0 moves the bytes.
  const unsigned long long mine = blockIdx.x < n_tasks ? (n_tasks - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
  unsigned long long my_src = 0, my_dst = 0;
  unsigned my_bytes = 0;
  unsigned long long slot_dst[kBulkStages];
  unsigned slot_bytes[kBulkStages];
  unsigned long long at = 0;                        // copies looked at
  unsigned head = 0, tail = 0;                      // loads issued, loads done with
  bool gave_up = false;
  for (;;) {
    // fill the ring: the slot of load `head` was last read by store head - kBulkStages, which is not the newest
    while (!gave_up && at < mine && head - tail < (tail ? kBulkStages - 1 : kBulkStages)) {
      if (at % 32 == 0) {
        my_bytes = 0;
        if (at + lane < mine) {
          const unsigned long long t = blockIdx.x + (at + lane) * gridDim.x, pp = t / pieces, piece = t - pp * pieces;
          const unsigned pool = static_cast<unsigned>(pp / n_pairs), pair = static_cast<unsigned>(pp - static_cast<unsigned long long>(pool) * n_pairs);
          const unsigned long long base = reinterpret_cast<unsigned long long>(FROM_ARRAY ? pools[pool] : two.p[pool]) + piece * kBulkBytes;
          const int src = __ldg(pairs + 2 * pair), dst = __ldg(pairs + 2 * pair + 1);
          my_src = base + static_cast<unsigned long long>(src) * block_bytes;
          my_dst = base + static_cast<unsigned long long>(dst) * block_bytes;
          my_bytes = src == dst ? 0u : static_cast<unsigned>(min(static_cast<unsigned long long>(kBulkBytes), block_bytes - piece * kBulkBytes));
        }
      }
      const unsigned long long src = __shfl_sync(0xffffffffu, my_src, static_cast<int>(at % 32)), dst = __shfl_sync(0xffffffffu, my_dst, static_cast<int>(at % 32));
      const unsigned bytes = __shfl_sync(0xffffffffu, my_bytes, static_cast<int>(at % 32));
      ++at;
      if (bytes == 0) continue;
      const unsigned slot = head % kBulkStages;
      if (lane == 0) {
        if (head >= kBulkStages) asm volatile("cp.async.bulk.wait_group.read 1;\n" ::: "memory");
        mbar_arrive_expect_tx(smem_u32(&full[slot]), bytes);
        bulk_load(smem_u32(ring) + slot * kBulkBytes, reinterpret_cast<const void*>(src), bytes, smem_u32(&full[slot]));
      }
#pragma unroll
      for (int i = 0; i < kBulkStages; ++i)
        if (i == static_cast<int>(slot)) { slot_dst[i] = dst; slot_bytes[i] = bytes; }
      ++head;
    }
    if (tail == head) break;
    const unsigned slot = tail % kBulkStages;
    // A wait that runs out ends the block's copies, but not before every load that is still on its way into the
    // ring has been waited for (as long again, once each) and those that arrive have been stored: the ring's memory
    // goes to another block when this one leaves.
    bool landed = mbar_wait(smem_u32(&full[slot]), (tail / kBulkStages) & 1u);
    landed = __all_sync(0xffffffffu, landed);
    if (!landed && !gave_up) {
      gave_up = true;
      if (lane == 0) copy_give_up(host_err);
      continue;
    }
    if (lane == 0 && landed) {
#pragma unroll
      for (int i = 0; i < kBulkStages; ++i)
        if (i == static_cast<int>(slot)) bulk_store(reinterpret_cast<void*>(slot_dst[i]), smem_u32(ring) + i * kBulkBytes, slot_bytes[i]);
    }
    ++tail;
    __syncwarp();
  }
  if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
}

// Blocks whose byte size or pool address is not 16-byte granular.
template <bool FROM_ARRAY>
__global__ void __launch_bounds__(kCopyThreads) copy_blocks_bytes_kernel(TwoPools two, void* const* __restrict__ pools,
                                                                          const int* __restrict__ pairs, size_t block_bytes) {
  char* pool = static_cast<char*>(FROM_ARRAY ? pools[blockIdx.z] : two.p[blockIdx.z]);
  const int src = pairs[2 * blockIdx.y], dst = pairs[2 * blockIdx.y + 1];
  if (src == dst) return;
  const char* s = pool + static_cast<size_t>(src) * block_bytes;
  char* d = pool + static_cast<size_t>(dst) * block_bytes;
  for (size_t i = blockIdx.x * static_cast<size_t>(kCopyThreads) + threadIdx.x; i < block_bytes;
       i += static_cast<size_t>(gridDim.x) * kCopyThreads)
    d[i] = s[i];
}

int copy_impl(TwoPools two, void* const* pools, int n_pools, bool pools_aligned, const int* pairs, int n_pairs,
              size_t block_bytes, pkv_stream stream) {
  if (n_pairs <= 0 || n_pools <= 0 || block_bytes == 0) return PKV_OK;
  if (!pairs) return fail(PKV_E_ARG, "pkv_copy_blocks: null pair list");
  if (n_pairs > 65535 || n_pools > 65535)
    return fail(PKV_E_UNSUPPORTED, "pkv_copy_blocks: at most 65535 pairs and 65535 pools per call (got %d, %d)", n_pairs, n_pools);
  const int st = check_error_mirror("pkv_copy_blocks", kErrCopyWait);   // a copy that gave up; anything else is the attention calls' to report
  if (st != PKV_OK) return st;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (block_bytes % 16 == 0 && pools_aligned) {
    const unsigned long long pieces = (block_bytes + kBulkBytes - 1) / kBulkBytes, tasks = pieces * n_pairs * n_pools;
    static thread_local int sms = 0;
    if (!sms) {
      int dev = 0;
      cudaGetDevice(&dev);
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      if (sms <= 0) sms = 148;
    }
    const unsigned blocks = static_cast<unsigned>(std::min<unsigned long long>(tasks, static_cast<unsigned long long>(sms) * kBulkBlocksPerSm));
    auto kern = pools ? copy_blocks_bulk_kernel<true> : copy_blocks_bulk_kernel<false>;
    unsigned int* mirror = error_mirror(true);
    launch_pdl(kern, dim3(blocks), dim3(32), kBulkStages * kBulkBytes, s, two, pools, pairs, n_pairs, block_bytes, pieces, tasks,
               mirror ? mirror + 1 : nullptr);               // the copies' own word
    return check_launch("copy_blocks_bulk_kernel");
  }
  dim3 grid(static_cast<unsigned>((block_bytes + kCopyThreads * 8 - 1) / (kCopyThreads * 8)), n_pairs, n_pools);
  if (pools) copy_blocks_bytes_kernel<true><<<grid, kCopyThreads, 0, s>>>(two, pools, pairs, block_bytes);
  else copy_blocks_bytes_kernel<false><<<grid, kCopyThreads, 0, s>>>(two, pools, pairs, block_bytes);
  return check_launch("copy_blocks_bytes_kernel");
}

int copy_two(void* k_cache, void* v_cache, const int* pairs, int n_pairs, int block_size, int kv_dim, size_t elem,
             pkv_stream stream) {
  if (n_pairs <= 0) return PKV_OK;
  if (!k_cache || !v_cache) return fail(PKV_E_ARG, "pkv_copy_blocks: null pool pointer");
  if (block_size <= 0 || kv_dim <= 0) return fail(PKV_E_ARG, "pkv_copy_blocks: block_size %d, kv_dim %d must be > 0", block_size, kv_dim);
  TwoPools two{{k_cache, v_cache}};
  return copy_impl(two, nullptr, 2, aligned16(k_cache) && aligned16(v_cache), pairs, n_pairs,
                   elem * static_cast<size_t>(block_size) * kv_dim, stream);
}

}  // namespace

// Reads and clears this file's share of the device error word (pkv_debug_device_flags).
int copy_read_flags(unsigned int* flags) {
  unsigned int v = 0, zero = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_pkv_copy_error, sizeof(v));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_pkv_copy_error, &zero, sizeof(zero));
  if (e != cudaSuccess) return fail(PKV_E_CUDA, "pkv_debug_device_flags: %s", cudaGetErrorString(e));
  *flags = v;
  return PKV_OK;
}
}  // namespace pkv

extern "C" {
int pkv_copy_blocks_f16(void* k_cache, void* v_cache, const int* src_dst_pairs, int n_pairs, int block_size,
                        int kv_dim, pkv_stream stream) {
  return pkv::copy_two(k_cache, v_cache, src_dst_pairs, n_pairs, block_size, kv_dim, 2, stream);
}
int pkv_copy_blocks_bf16(void* k_cache, void* v_cache, const int* src_dst_pairs, int n_pairs, int block_size,
                         int kv_dim, pkv_stream stream) {
  return pkv::copy_two(k_cache, v_cache, src_dst_pairs, n_pairs, block_size, kv_dim, 2, stream);
}
int pkv_copy_blocks_f32(void* k_cache, void* v_cache, const int* src_dst_pairs, int n_pairs, int block_size,
                        int kv_dim, pkv_stream stream) {
  return pkv::copy_two(k_cache, v_cache, src_dst_pairs, n_pairs, block_size, kv_dim, 4, stream);
}
// The pool base pointers live in device memory, so their alignment cannot be
// inspected here: every pool must be 16-byte aligned when block_bytes is a
// multiple of 16 (cudaMalloc'd pools always are).
int pkv_copy_blocks_layers(void* const* d_cache_ptrs, int n_caches, const int* src_dst_pairs, int n_pairs,
                           size_t block_bytes, pkv_stream stream) {
  if (n_pairs <= 0 || n_caches <= 0) return PKV_OK;
  if (!d_cache_ptrs) return pkv::fail(PKV_E_ARG, "pkv_copy_blocks_layers: null pool pointer array");
  pkv::TwoPools two{{nullptr, nullptr}};
  return pkv::copy_impl(two, d_cache_ptrs, n_caches, true, src_dst_pairs, n_pairs, block_bytes, stream);
}
}
