// Shared device helpers for the paged-KV kernels (sm_100a).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace pkv {

// ---- element traits ---------------------------------------------------------
template <typename T> struct Elem;
template <> struct Elem<float> {
  static __device__ __forceinline__ float to_f32(float x) { return x; }
  static __device__ __forceinline__ float from_f32(float x) { return x; }
};
template <> struct Elem<__half> {
  static __device__ __forceinline__ float to_f32(__half x) { return __half2float(x); }
  static __device__ __forceinline__ __half from_f32(float x) { return __float2half_rn(x); }
};
template <> struct Elem<__nv_bfloat16> {
  static __device__ __forceinline__ float to_f32(__nv_bfloat16 x) { return __bfloat162float(x); }
  static __device__ __forceinline__ __nv_bfloat16 from_f32(float x) { return __float2bfloat16_rn(x); }
};

// Two fp32 values -> one 32-bit register of two 16-bit floats (lo in the low half).
template <typename T> __device__ __forceinline__ uint32_t pack2(float lo, float hi);
template <> __device__ __forceinline__ uint32_t pack2<__half>(float lo, float hi) {
  __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}
template <> __device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float lo, float hi) {
  __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}

// ---- asynchronous global -> shared copies (LDGSTS) ------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// 16-byte copy that bypasses L1; src_bytes == 0 writes zeros instead of reading.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// ---- warp-level matrix fragments ----------------------------------------------
__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}

// D(16x8, f32) += A(16x16) * B(16x8), 16-bit inputs.
template <typename T> __device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1);
template <> __device__ __forceinline__ void mma16816<__half>(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <> __device__ __forceinline__ void mma16816<__nv_bfloat16>(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// ---- cache-hinted loads ---------------------------------------------------------
__device__ __forceinline__ uint4 ld_nc_u4(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

// ---- integer scans -----------------------------------------------------------------
struct ScanSum { static __device__ __forceinline__ int op(int a, int b) { return a + b; } };
struct ScanMax { static __device__ __forceinline__ int op(int a, int b) { return max(a, b); } };
template <typename Op>
__device__ __forceinline__ int warp_scan(int v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v = Op::op(v, x);
  }
  return v;
}
// Inclusive scan over a block of WARPS full warps, one value per thread.  `sm` holds one word per warp and is
// free for the next scan only after another barrier; *total receives the block's result.
template <typename Op, int WARPS>
__device__ __forceinline__ int block_scan(int v, int* sm, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = warp_scan<Op>(v, lane);
  if (lane == 31) sm[warp] = v;
  __syncthreads();
  const int w = warp_scan<Op>(sm[min(lane, WARPS - 1)], lane);   // every warp scans the totals for itself: one barrier
  const int before = __shfl_sync(0xffffffffu, w, max(warp - 1, 0));
  *total = __shfl_sync(0xffffffffu, w, WARPS - 1);
  return warp ? Op::op(before, v) : v;
}

// ---- runs of a packed step ---------------------------------------------------------
// A run is a maximal stretch of packed tokens of one sequence at consecutive positions.  Called by every thread
// of a block of WARPS warps for n <= PER * 32 WARPS tokens; each thread gets PER consecutive tokens from
// tid * ceil(n / threads), fewer at the end (first, count), with their positions, sequences and run lengths;
// start_of holds the first token of each one's run.  pos, seq and scratch are shared-memory arrays of n words, `sm`
// one of WARPS; ends without a barrier (the arrays may be reused after one).
template <int WARPS, int PER> struct TokenRuns {
  int first, count;
  int pos[PER], seq[PER], start_of[PER], len[PER];
  __device__ __forceinline__ void find(const int* __restrict__ token_pos, const int* __restrict__ token_seq, int n, int* s_pos,
                                       int* s_seq, int* scratch, int* sm) {
    constexpr int kThreads = 32 * WARPS;
    for (int t = threadIdx.x; t < n; t += kThreads) {
      s_pos[t] = token_pos[t];
      s_seq[t] = token_seq[t];
    }
    __syncthreads();
    const int per = (n + kThreads - 1) / kThreads;
    first = threadIdx.x * per;
    count = max(0, min(per, n - first));
    auto starts = [&](int t) { return t == 0 || s_seq[t - 1] != s_seq[t] || s_pos[t - 1] + 1 != s_pos[t]; };
    int last = -1;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      pos[i] = 0; seq[i] = 0; start_of[i] = -1; len[i] = 0;
      if (i < count) {
        pos[i] = s_pos[first + i];
        seq[i] = s_seq[first + i];
        if (starts(first + i)) last = first + i;
        start_of[i] = last;
      }
    }
    int total;
    const int upto = block_scan<ScanMax, WARPS>(last, sm, &total);
    int before = __shfl_up_sync(0xffffffffu, upto, 1);
    if ((threadIdx.x & 31) == 0) {                       // the inclusive result of the warp before
      before = -1;
      for (int w = 0; w < static_cast<int>(threadIdx.x >> 5); ++w) before = max(before, sm[w]);
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      if (i < count) {
        if (start_of[i] < 0) start_of[i] = before;
        const int t = first + i;
        if (t == n - 1 || starts(t + 1)) scratch[start_of[i]] = t - start_of[i] + 1;
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (i < count) len[i] = scratch[start_of[i]];
  }
};

__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

}  // namespace pkv
