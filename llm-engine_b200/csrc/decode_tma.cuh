// Paged decode attention, TMA variant (sm_100a): head_dim 64 or 128, block_size a multiple
// of 16, 16-bit K/V with a GQA group of up to 16 or fp32 K/V with one of up to 8.
//
// Work unit = (token, key range) x kv head.  Every WARP is an independent worker:
// it owns a private ring of shared-memory stages, fetches its own units, and
// finishes them on its own -- there is no block-wide barrier and no cross-warp
// merge anywhere in the kernel, so the look-ups at the start of a unit and the
// store / split-K arrival at its end stall one warp out of the twelve or sixteen on
// the SM while the others keep the memory system busy.
//
//   loads   one lane issues TMA box copies (cp.async.bulk.tensor.2d: 16 slots x 128
//           bytes, 128-byte swizzle) through the block table, one box per 16 keys for
//           K and for V, completing on the stage's mbarrier.  The issue pointer runs
//           NSTAGES slabs ahead of the math and crosses unit boundaries, so the ring
//           never drains between units.  Table entries are fetched 32 boxes at a
//           time (one coalesced load) and handed out by shuffle.
//   math    keys are the M dimension of mma.sync m16n8k16 and the group's query heads
//           the N dimension (S^T = K Q^T, O^T = V^T P^T): a group of up to 8 heads
//           wastes no tensor-core rows, and the online-softmax state of a head lives
//           in the thread that owns its accumulator column -- no cross-lane traffic
//           for the rescale, three shuffles per slab for the running maximum, one
//           movmatrix per 8x8 block of P.
//           fp32 K/V: fp32 arithmetic throughout (packed fused multiply-adds), see there.
//   finish  a unit that covers its token's whole history writes the output rows; any
//           other writes its split-K partial, fire and forget; decode_combine_kernel
//           (decode_attn.cuh) merges the partials afterwards.
//
// Every mbarrier wait is bounded; a wait that runs out records a flag (device word and the
// host's pinned word) and the warp winds down instead of spinning.  Blocks are persistent and all
// start together, so a launch ends within a few wait limits whatever happens; a recorded flag
// does not stop later launches.
#pragma once

#include "decode_attn.cuh"
#include "tma_util.hpp"

namespace pkv {

constexpr unsigned kErrProducerWait = 1u, kErrConsumerWait = 2u;

constexpr int kBoxBytes = 16 * 128;

struct WarpGroup {
  static __device__ __forceinline__ void sync() { __syncwarp(); }
  static __device__ __forceinline__ int size() { return 32; }
  static __device__ __forceinline__ int tid() { return threadIdx.x & 31; }
};

template <int D, int MT, int NSTAGES, int WARPS, int ELEM = 2> struct TmaSmem {
  static constexpr int kHalves = D * ELEM / 128;             // 128-byte boxes side by side in a row
  static constexpr int kKBytes = MT * kHalves * kBoxBytes;  // K part of a stage; V follows
  static constexpr int kStageBytes = 2 * kKBytes;
  static constexpr int kWarpBytes = NSTAGES * kStageBytes;
  static constexpr int kQBytes = ELEM == 4 ? 8 * (D + 4) * 4 : 0;   // fp32: a warp's query rows, behind the rings
  static constexpr int kBytes = WARPS * (kWarpBytes + kQBytes) + 1024;
};

// TOK = 1: a unit serves one token.  TOK = 4: a unit serves up to four tokens whose sequences
// share the blocks of its key range (a common prompt prefix): the K/V slab is fetched once and
// the tokens' heads sit side by side in the N dimension (NT / TOK head tiles per token); every
// token gets its own split-K partial.  Such units come from the shared-prefix planner as
// SharedItem records (decode_plan.hpp).
// FUSED_APPEND: the unit that reaches a token's newest key takes that row from the step's k / v
// inputs and writes it to the pool (DecodeArgs::new_k); a separate instantiation, so that the
// plain kernel carries none of it.
// CLUSTER: small steps.  The launch is a grid of thread-block clusters, one cluster per (token, kv
// head); the history is cut into as many equal ranges as the cluster has warps (fewer when it is
// short), warp w of block r takes range w * blocks + r, and the split-K merge happens inside the
// launch.  Block r of the cluster owns query heads r, r + blocks, ... of the group: a warp that has
// finished its range sends, for every head, that head's 64 sums and (maximum, sum) to the head's
// owner -- st.async stores into the owner's landing area in shared memory, each completing bytes
// on the owner's mbarrier -- and every block, once its barrier has counted all the bytes its heads
// expect, folds them from its own shared memory into the output rows.  No plan, no workspace, no
// merge kernel, no cluster-wide barrier after the first (which only publishes the mbarriers): the
// ranges and the byte counts follow from token_pos alone.
__host__ __device__ constexpr int cluster_record(int d) { return (d + 4) * 4; }   // one (head, range) record in a landing area: d sums, maximum, sum, 8 bytes unused
// Landing area of a block: records for ceil(8 / blocks) heads x (4 warps x blocks) ranges; the
// cluster sizes the launcher offers (2, 3, 4, 8) need at most 3 x 12 of them.
__host__ __device__ constexpr int cluster_land_bytes(int d) { return 36 * cluster_record(d) + 96; }
__host__ __device__ constexpr bool cluster_size_ok(int cs) { return cs == 2 || cs == 3 || cs == 4 || cs == 8; }

__device__ __forceinline__ uint32_t cluster_map(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
// 16 bytes into another block's shared memory; the bytes count on that block's mbarrier when they land.
__device__ __forceinline__ void cluster_push4(uint32_t dst_cluster_addr, float4 v, uint32_t bar_cluster_addr) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];\n" ::"r"(dst_cluster_addr),
               "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(bar_cluster_addr)
               : "memory");
}

// Place in a warp's list of units: (item, kv head), with `end` the end of the items of the current share.
struct UnitCursor { int u, item, end, kvh; };

// A step's plan in shared memory, built by every block for itself (DecodeArgs::inline_min_run): the same cuts
// as decode_plan_kernel makes, found through the tokens instead of a list.  A planner launch in front of the
// attention kernel cost 4.6 us a layer, and the four dependent look-ups from its list to a unit's first load
// 2 to 3 more; this takes every block about 4 (16 us a layer without the planner launch, 19 with it, 48 sequences).
struct InlinePlan {
  static constexpr int kPer = (kInlineTokens + 127) / 128;
  static constexpr int kBytes = kInlineTokens * (3 * 4 + 2);
  struct Unit { int token, begin, len, part; };
  int* s_len;              // keys of a token the decode path handles: position + 1, or 0
  int* s_tbl;              // where its block table starts
  int* s_key;              // shares: where it begins in the laid-out step, in slabs; chunks: its first item
  unsigned short* s_part;  // its first partial slot
  ShareRule rule;
  int n_items;

  __device__ __forceinline__ int table_of(int token) const { return s_tbl[token]; }

  __device__ __forceinline__ void build(const DecodeArgs& a, unsigned char* smem) {
    __shared__ int sm_scan[3][4];
    __shared__ int sm_step[2];                                             // longest token, whether there is a run for the prefill kernel
    if (threadIdx.x < 2) sm_step[threadIdx.x] = 0;                         // (the barriers of find() come before its first use)
    s_len = reinterpret_cast<int*>(smem);
    s_tbl = s_len + kInlineTokens;
    s_key = s_tbl + kInlineTokens;
    s_part = reinterpret_cast<unsigned short*>(s_key + kInlineTokens);
    const int n = a.n_tokens;
    TokenRuns<4, kPer> runs;
    runs.find(a.token_pos, a.token_seq, n, s_len, s_tbl, s_key, sm_scan[0]);
    int len[kPer], tbl[kPer], slabs = 0, longest = 0;
    bool in_run = false;
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      len[i] = tbl[i] = 0;
      in_run |= i < runs.count && runs.len[i] >= a.inline_min_run;
      if (i < runs.count && runs.len[i] < a.inline_min_run) {
        len[i] = max(runs.pos[i], 0) + 1;
        tbl[i] = __ldg(a.table_offset + runs.seq[i]);
        slabs += share_padded(len[i]) / kShareSlab;
        longest = max(longest, len[i]);
      }
    }
    longest = __reduce_max_sync(0xffffffffu, longest);
    if ((threadIdx.x & 31) == 0) atomicMax(&sm_step[0], longest);
    if (in_run) sm_step[1] = 1;
    int total;
    int at = block_scan<ScanSum, 4>(slabs, sm_scan[1], &total) - slabs;    // (and the barrier after which the arrays are free)
    rule = ordered_share_rule(total, sm_step[0], a.inline_max_shares, sm_step[1] == 0);
    int begin[kPer], ns[kPer], sum = 0;                                    // items in the upper half, partials in the lower: < 2^16 each
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      begin[i] = at;
      ns[i] = 0;
      if (len[i] > 0) {
        const int padded = share_padded(len[i]);
        ns[i] = rule.per > 0 ? share_cuts(static_cast<long long>(at) * kShareSlab, padded, rule.per).n + 1
                             : rule.chunk > 0 ? (len[i] + rule.chunk - 1) / rule.chunk : 1;
        at += padded / kShareSlab;
      }
      sum += (ns[i] << 16) | (ns[i] > 1 ? ns[i] : 0);
    }
    int all;
    int before = block_scan<ScanSum, 4>(sum, sm_scan[2], &all) - sum;
    n_items = all >> 16;
    TokSplit* split = const_cast<TokSplit*>(a.tok_split);
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      if (i < runs.count) {
        const int t = runs.first + i;
        s_len[t] = len[i];
        s_tbl[t] = tbl[i];
        s_key[t] = rule.per > 0 ? begin[i] : before >> 16;
        s_part[t] = static_cast<unsigned short>(before & 0xffff);
        if (blockIdx.x == 0) split[t] = TokSplit{before & 0xffff, ns[i]};
        before += (ns[i] << 16) | (ns[i] > 1 ? ns[i] : 0);
      }
    }
    __syncthreads();
  }

  // How many tokens have s_key < v (they come first: s_key does not decrease); by the whole warp.
  __device__ __forceinline__ int below(int v, int n) const {
    const int lane = threadIdx.x & 31, step = (n + 31) / 32;               // <= 22
    const int last = (lane + 1) * step - 1;
    const int seg = __popc(__ballot_sync(0xffffffffu, last < n && s_key[min(last, n - 1)] < v));
    const int i = seg * step + lane;
    return seg * step + __popc(__ballot_sync(0xffffffffu, lane < step && i < n && s_key[min(i, n - 1)] < v));
  }

  // The next unit of the warp's list; x.end: 1 while inside a share, whose next token is x.item.
  __device__ __forceinline__ bool next(UnitCursor& x, Unit& w, int total, int stride, int kv_heads, int n) const {
    if (rule.per == 0) {
      x.u += stride;
      if (x.u >= total) { x.u = total; return false; }
      const int item = x.u / kv_heads;
      x.kvh = x.u - item * kv_heads;
      const int t = below(item + 1, n) - 1;                                // the last token whose first item is not past this one
      const int len = s_len[t], s = item - s_key[t];
      w.token = t;
      w.begin = s * rule.chunk;
      w.len = rule.chunk > 0 ? min(rule.chunk, len - w.begin) : len;
      w.part = w.len < len ? s_part[t] + s : -1;
      return true;
    }
    const int per = rule.per / kShareSlab;                                 // all in slabs from here
    for (;;) {
      if (x.end == 0) {
        x.u += stride;
        if (x.u >= total) { x.u = total; return false; }
        const int j = x.u / kv_heads, c = j * per;
        x.kvh = x.u - j * kv_heads;
        x.item = below(c - 1, n);                                          // the first token that begins in this share
        x.end = 1;
        const int t = x.item - 1;
        if (t >= 0) {
          const int b = s_key[t], e = b + share_padded(s_len[t]) / kShareSlab;
          if (e - c > 1) {                                                 // the token before it is cut here
            const bool again = e - (c + per) > 1;
            w.token = t;
            w.begin = (c - b) * kShareSlab;
            w.len = again ? rule.per : s_len[t] - w.begin;
            w.part = s_part[t] + (c - ((b + 1) / per + 1) * per) / per + 1;
            if (again) x.end = 0;
            return true;
          }
        }
      }
      const int j = x.u / kv_heads;
      int t = x.item;
      if (t < n && s_len[t] == 0) t = below(s_key[t] + 1, n) - 1;          // tokens of long runs begin where the next token does
      if (t >= n || s_len[t] == 0 || min((s_key[t] + 1) / per, rule.n_shares - 1) > j) { x.end = 0; continue; }
      const int b = s_key[t], e = b + share_padded(s_len[t]) / kShareSlab, cut = ((b + 1) / per + 1) * per;
      const bool cuts = e - cut > 1;
      w.token = t;
      w.begin = 0;
      w.len = cuts ? (cut - b) * kShareSlab : s_len[t];
      w.part = cuts ? s_part[t] : -1;
      x.item = t + 1;
      if (cuts) x.end = 0;
      return true;
    }
  }
};

// (a.x, a.y) * (b.x, b.y) + (c.x, c.y), each rounded once, in one instruction.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n .reg .b64 ra, rb, rc, rd;\n mov.b64 ra, {%2, %3};\n mov.b64 rb, {%4, %5};\n mov.b64 rc, {%6, %7};\n"
      " fma.rn.f32x2 rd, ra, rb, rc;\n mov.b64 {%0, %1}, rd;\n}\n"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}

template <typename T, int D, int NT, int MT, int NSTAGES, int WARPS, int MIN_BLOCKS, int TOK = 1, bool FUSED_APPEND = false,
          bool CLUSTER = false, bool INLINE_PLAN = false>
__global__ void __launch_bounds__(WARPS * 32, MIN_BLOCKS)
    decode_tma_kernel(const DecodeArgs a, const __grid_constant__ CUtensorMap kmap,
                      const __grid_constant__ CUtensorMap vmap) {
  using S = TmaSmem<D, MT, NSTAGES, WARPS, sizeof(T)>;
  constexpr bool F32 = sizeof(T) == 4;
  static_assert(!F32 || (NT == 1 && MT == 1 && TOK == 1 && !FUSED_APPEND), "fp32: up to 8 heads, slabs of 16 keys");
  static_assert(TOK == 1 || TOK == 4, "a shared unit holds four tokens");
  static_assert(NT % TOK == 0, "whole head tiles per token");
  static_assert(!CLUSTER || TOK == 1, "cluster launches take ordinary tokens");
  static_assert(!CLUSTER || NT == 1, "the cluster form is written for up to 8 heads per kv head");
  constexpr int kClusterRecord = cluster_record(D);
  static_assert(!CLUSTER || (8 * NT * D + 32 * NT) * 4 <= S::kWarpBytes, "a warp's partial must fit its ring");
  constexpr int NTG = NT / TOK;   // head tiles (8 heads each) per token
  constexpr int KS = D / 16;
  constexpr int HALVES = S::kHalves;
  constexpr int SLAB = 16 * MT;
  constexpr int kBoxCols = 128 / static_cast<int>(sizeof(T));
  constexpr float kLog2e = 1.4426950408889634f;

  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long full_bar[WARPS * NSTAGES];
  __shared__ __align__(8) unsigned long long land_bar;     // cluster launches: counts the bytes this block's heads expect

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, c = lane & 3;
  const uint32_t ring0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t ring = ring0 + warp * S::kWarpBytes;
  unsigned char* ring_ptr = smem_raw + (ring - smem_u32(smem_raw));
  const uint32_t bars = smem_u32(&full_bar[warp * NSTAGES]);
  const float sl2 = a.scale * kLog2e;

  if (lane == 0) {
#pragma unroll
    for (int s = 0; s < NSTAGES; ++s) mbar_init(bars + 8 * s, 1);
    mbar_fence_init();
  }
  __syncwarp();

  // Everything above touched only this block's shared memory.  What follows reads the plan and the
  // step's index arrays, which are complete before the predecessor on the stream even starts (they
  // are built once per step, ahead of every layer's launches, by copies or by kernels that do not
  // release their dependents early), so the look-ups that lead to a unit's first load -- item, sequence,
  // table offset, table entries -- run while the predecessor is still finishing.  What the predecessor
  // itself may have written (pool rows appended by the preceding launch, q and the new k / v rows, the
  // workspace the previous merge has finished with) is touched only after griddepcontrol.wait, which
  // every lane executes in issue_next() right before the warp's first load is issued -- or, with the
  // append inside this launch, only before the unit's q rows are read (see there): the pool rows it
  // loads are then all from earlier steps.
  pdl_launch_dependents();
  if (lane == 0) {
    asm volatile("prefetch.tensormap [%0];\n" ::"l"(&kmap) : "memory");
    asm volatile("prefetch.tensormap [%0];\n" ::"l"(&vmap) : "memory");
  }
  bool waited = !CLUSTER && !FUSED_APPEND && a.wait_last != 0;
  // Cluster launches: this warp's one unit, from the token's position alone (a step constant).
  int c_token = 0, c_kvh = 0, c_begin = 0, c_len = 0, c_nsplits = 1, c_split = 0;
  uint32_t c_rank = 0, c_size = 1;
  if constexpr (CLUSTER) {
    asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(c_rank));
    asm volatile("mov.u32 %0, %%cluster_nctarank;\n" : "=r"(c_size));
    const int pair = blockIdx.x / c_size;                  // clusters are runs of consecutive blocks
    c_token = pair / a.kv_heads;
    c_kvh = pair - c_token * a.kv_heads;
    const int len = max(__ldg(a.token_pos + c_token), 0) + 1;
    const int nw = WARPS * static_cast<int>(c_size);
    const int range = (((len + nw - 1) / nw + SLAB - 1) / SLAB) * SLAB;   // whole slabs per warp
    c_nsplits = (len + range - 1) / range;
    c_split = warp * static_cast<int>(c_size) + static_cast<int>(c_rank);   // neighbouring ranges on different SMs
    c_begin = c_split * range;
    c_len = min(range, len - c_begin);                     // <= 0: no unit for this warp
    if (c_nsplits > 1) {                                   // the same for every thread of the cluster
      if (threadIdx.x == 0) {
        const int owned = (a.group - static_cast<int>(c_rank) + static_cast<int>(c_size) - 1) / static_cast<int>(c_size);
        mbar_init(smem_u32(&land_bar), 1);
        mbar_fence_init();
        // all of this block's heads' records, from every range; a block that owns no head (fewer heads
        // than blocks) expects nothing and its barrier completes at once
        mbar_arrive_expect_tx(smem_u32(&land_bar), static_cast<uint32_t>(owned * c_nsplits * kClusterRecord));
      }
      // publish the barriers: nobody sends before every block has armed its own (waited for below,
      // right before the first send, by which time it has long completed)
      __syncwarp();
      asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    }
  }
  // Units of this warp: one item each (item, kv head) dealt round-robin, or, when the plan has shares, all the
  // items of a (share, kv head) one after the other.  The issue side and the math side walk the same list,
  // each with a cursor of its own.
  static_assert(!INLINE_PLAN || (TOK == 1 && !FUSED_APPEND && !CLUSTER && !F32 && WARPS == 4), "16-bit calls without a plan of the caller's");
  InlinePlan ip = {};
  if constexpr (INLINE_PLAN) {
    if (!waited) {       // not behind a prefill launch that has waited for the index arrays' producers
      pdl_wait();
      waited = true;
    }
    ip.build(a, smem_raw + (ring0 - smem_u32(smem_raw)) + WARPS * S::kWarpBytes);
  }
  const int n_shares = INLINE_PLAN ? ip.rule.n_shares : (CLUSTER || TOK > 1 || a.direct) ? 0 : a.header->n_shares;
  const int n_items = INLINE_PLAN ? ip.n_items : CLUSTER ? 0 : (TOK > 1 ? a.n_shared : (a.direct ? a.n_tokens : a.header->n_items));
  const int total = CLUSTER ? (c_len > 0 ? 1 : 0) : (n_shares > 0 ? n_shares : n_items) * a.kv_heads;
  const int gw = CLUSTER ? 0 : blockIdx.x * WARPS + warp, GW = CLUSTER ? 1 : gridDim.x * WARPS;
  const int* share_first = CLUSTER || TOK > 1 || INLINE_PLAN || a.direct ? nullptr : reinterpret_cast<const int*>(a.items + n_items);
  using Cursor = UnitCursor;
  auto next_unit = [&](Cursor& x) -> bool {
    if constexpr (CLUSTER) {             // at most one unit
      x.kvh = c_kvh;
      return ++x.u < total;
    }
    ++x.item;
    while (x.item >= x.end) {
      x.u += GW;
      if (x.u >= total) { x.u = total; x.item = x.end = 0; return false; }
      x.item = x.u / a.kv_heads;
      x.kvh = x.u - x.item * a.kv_heads;
      x.end = x.item + 1;
      if (n_shares > 0) {
        x.end = __ldg(share_first + x.item + 1);
        x.item = __ldg(share_first + x.item);
      }
    }
    return true;
  };

  // ---------------------------- issue side ----------------------------
  Cursor ic{gw - GW, 0, 0, 0};  // unit the issue pointer is in (advanced before first use)
  int i_nslabs = 0, i_slab = 0, i_kvbeg = 0, i_len = 0, i_x0 = 0;
  const int* i_tbl = nullptr;
  int i_ent = 0, i_ent_base = -64;   // this lane's block-table entry for box i_ent_base + lane
  uint32_t n_issued = 0, n_consumed = 0;

  InlinePlan::Unit i_unit, m_unit;
  // Issues the next slab of this warp's unit sequence, if there is one.
  auto issue_next = [&]() -> bool {
    while (i_slab >= i_nslabs) {
      if (!(INLINE_PLAN ? ip.next(ic, i_unit, total, GW, a.kv_heads, a.n_tokens) : next_unit(ic))) return false;
      const int item = ic.item, kvh = ic.kvh;
      int token, part;
      if constexpr (INLINE_PLAN) {
        token = i_unit.token;
        i_kvbeg = i_unit.begin;
        i_len = i_unit.len;
        part = 0;
      } else if constexpr (CLUSTER) {
        token = c_token;
        i_kvbeg = c_begin;
        i_len = c_len;
        part = 0;
      } else if constexpr (TOK > 1) {
        const int4 h0 = __ldg(a.shared_items + 3 * item), tk = __ldg(a.shared_items + 3 * item + 1);
        i_kvbeg = h0.x;
        i_len = h0.y;
        token = tk.x;          // every token of the unit has the same blocks over this range
        part = 0;
      } else {
        load_item(a, item, token, i_kvbeg, i_len, part);
      }
      if constexpr (INLINE_PLAN) i_tbl = a.block_tables + ip.table_of(token);
      else i_tbl = a.block_tables + __ldg(a.table_offset + __ldg(a.token_seq + token));
      i_nslabs = (i_len + SLAB - 1) / SLAB;
      i_slab = 0;
      i_x0 = kvh * D;
      i_ent_base = -64;
      // warm the query rows of this unit for the math side (group x D 16-bit values)
      if constexpr (TOK == 1) {
        const char* qrow = reinterpret_cast<const char*>(static_cast<const T*>(a.q) +
                                                         (static_cast<size_t>(token) * a.q_heads + kvh * a.group) * D);
        if (lane * 128 < a.group * D * static_cast<int>(sizeof(T))) asm volatile("prefetch.global.L2 [%0];\n" ::"l"(qrow + lane * 128));
      }
    }
    const int box0 = i_slab * MT;
    if (box0 + MT > i_ent_base + 32) {   // fetch the entries of the next 32 boxes in one coalesced load
      i_ent_base = box0;
      const int rel = (box0 + lane) * 16;
      i_ent = rel < i_len ? __ldg(i_tbl + ((i_kvbeg + rel) >> a.bs_log2)) : 0;
    }
    int ent[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) ent[m] = __shfl_sync(0xffffffffu, i_ent, box0 + m - i_ent_base);
    if constexpr (!FUSED_APPEND) {
      if (!waited) {
        pdl_wait();
        waited = true;
      }
    }
    // The slot's previous contents were read with ordinary loads (ldmatrix) by all
    // lanes; order those before the asynchronous-proxy write that refills it.
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncwarp();
    if (lane == 0) {
      const uint32_t slot = n_issued % NSTAGES;
      const uint32_t fb = bars + 8 * slot;
      const uint32_t st = ring + slot * S::kStageBytes;
      const int rel0 = i_slab * SLAB;
      int nvalid = 0;
#pragma unroll
      for (int m = 0; m < MT; ++m) nvalid += (rel0 + 16 * m < i_len) ? 1 : 0;
      mbar_arrive_expect_tx(fb, static_cast<uint32_t>(nvalid) * 2u * HALVES * kBoxBytes);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        if (rel0 + 16 * m < i_len) {
          const int key0 = i_kvbeg + rel0 + 16 * m;
          const int y = (ent[m] << a.bs_log2) + (key0 & (a.block_size - 1));
#pragma unroll
          for (int h = 0; h < HALVES; ++h) {
            const uint32_t dst = st + (m * HALVES + h) * kBoxBytes;
            tma_load_2d(dst, &kmap, i_x0 + kBoxCols * h, y, fb);
            tma_load_2d(dst + S::kKBytes, &vmap, i_x0 + kBoxCols * h, y, fb);
          }
        }
      }
    }
    ++n_issued;
    ++i_slab;
    return true;
  };

  // ---------------------------- math side -----------------------------
  const int mi = lane >> 3, r8 = lane & 7;
  bool more = true;
  Cursor mc{gw - GW, 0, 0, 0};
  while (INLINE_PLAN ? ip.next(mc, m_unit, total, GW, a.kv_heads, a.n_tokens) : next_unit(mc)) {
    const int item = mc.item, kvh = mc.kvh;
    int token, kv_begin, kv_len, part;
    int toks[TOK], parts[TOK], n_tok = 1;
    if constexpr (INLINE_PLAN) {
      token = m_unit.token; kv_begin = m_unit.begin; kv_len = m_unit.len; part = m_unit.part;
      toks[0] = token; parts[0] = part;
    } else if constexpr (CLUSTER) {
      token = c_token; kv_begin = c_begin; kv_len = c_len;
      part = c_nsplits > 1 ? c_split : -1;
      toks[0] = token; parts[0] = part;
    } else if constexpr (TOK > 1) {
      const int4 h0 = __ldg(a.shared_items + 3 * item), tk = __ldg(a.shared_items + 3 * item + 1),
                 pt = __ldg(a.shared_items + 3 * item + 2);
      kv_begin = h0.x; kv_len = h0.y; n_tok = h0.z;
      toks[0] = tk.x; toks[1] = tk.y; toks[2] = tk.z; toks[3] = tk.w;
      parts[0] = pt.x; parts[1] = pt.y; parts[2] = pt.z; parts[3] = pt.w;
      token = toks[0]; part = parts[0];
    } else {
      load_item(a, item, token, kv_begin, kv_len, part);
      toks[0] = token; parts[0] = part;
    }
    const int n_slabs = (kv_len + SLAB - 1) / SLAB;

    while (more && n_issued - n_consumed < NSTAGES) more = issue_next();

    if constexpr (FUSED_APPEND) {
      // With the append inside this launch the loads issued above fetch only rows of EARLIER steps (the
      // newest row comes from the step's k / v below): they need not wait for the predecessor, which
      // cannot be writing them -- a step's launches are preceded by that step's uploads or planning,
      // which complete before anything behind them starts.  What the predecessor does produce -- q, the
      // new k / v rows -- and everything this launch writes comes after this wait.
      if (!waited) {
        pdl_wait();
        waited = true;
      }
    }
    // Q^T fragments (B operand): rows = dims, columns = heads of the group.
    uint32_t qb[KS][NT][2];
    if constexpr (!F32) {
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const int ti = nt / NTG;                    // which token of the unit this head tile belongs to
        const T* qbase = static_cast<const T*>(a.q) + (static_cast<size_t>(toks[ti]) * a.q_heads + kvh * a.group) * D;
        const int head = 8 * (nt % NTG) + g;
        const bool hv = head < a.group && ti < n_tok;
        const uint32_t* qrow = reinterpret_cast<const uint32_t*>(qbase + static_cast<size_t>(head) * D);
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
          qb[ks][nt][0] = hv ? __ldg(qrow + ks * 8 + c) : 0u;
          qb[ks][nt][1] = hv ? __ldg(qrow + ks * 8 + 4 + c) : 0u;
        }
      }
    }
    float o[KS][NT][4];
    float m_run[NT][2], l_run[NT][2];
    // fp32: lane = (half of the dims, key of the slab) for the scores, whose running maximum and (this
    // key's share of the) sum it keeps for four heads, and = 2 or 4 dims of all eight heads for the sums.
    const int f_key = lane & 15, f_part = lane >> 4;
    float f_m[4], f_l[4];
    float2 f_o[8][D / 64];
    float* f_q = reinterpret_cast<float*>(ring_ptr + (WARPS - warp) * S::kWarpBytes + warp * S::kQBytes);
    if constexpr (F32) {
#pragma unroll
      for (int i = 0; i < 4; ++i) { f_m[i] = -INFINITY; f_l[i] = 0.f; }
#pragma unroll
      for (int h = 0; h < 8; ++h)
#pragma unroll
        for (int x = 0; x < D / 64; ++x) f_o[h][x] = make_float2(0.f, 0.f);
      // query rows, zeros past the group; the upper half of a row sits 16 bytes further on, so that the two
      // halves of the warp read different banks
      __syncwarp();
      for (int i = lane; i < 8 * (D / 4); i += 32) {
        const int h = i / (D / 4), d = 4 * (i - h * (D / 4));
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (h < a.group) x = __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(a.q) + (static_cast<size_t>(token) * a.q_heads + kvh * a.group + h) * D + d));
        *reinterpret_cast<float4*>(f_q + h * (D + 4) + d + (d >= D / 2 ? 4 : 0)) = x;
      }
      __syncwarp();
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      m_run[nt][0] = m_run[nt][1] = -INFINITY;
      l_run[nt][0] = l_run[nt][1] = 0.f;
#pragma unroll
      for (int dm = 0; dm < KS; ++dm) o[dm][nt][0] = o[dm][nt][1] = o[dm][nt][2] = o[dm][nt][3] = 0.f;
    }

    bool ok = true;
    for (int j = 0; j < n_slabs; ++j) {
      while (more && n_issued - n_consumed < NSTAGES) more = issue_next();
      const uint32_t slot = n_consumed % NSTAGES;
      if (!mbar_wait(bars + 8 * slot, (n_consumed / NSTAGES) & 1u)) {
        if (lane == 0) report_give_up(a, kErrConsumerWait);
        ok = false;
        break;
      }
      const uint32_t kst = ring + slot * S::kStageBytes;
      const uint32_t vst = kst + S::kKBytes;
      const int rows_valid = min(SLAB, kv_len - j * SLAB);
      if constexpr (TOK == 1 && FUSED_APPEND) {
        if (j == n_slabs - 1 && kv_begin + kv_len == __ldg(a.token_pos + token) + 1) {
          // Fused append: this unit ends at the token's newest key, whose row is not in the pool yet.
          // Lanes 0 .. 8 HALVES - 1 bring the 16-byte pieces of its K row, the next 8 HALVES those of
          // its V row: each goes into the slab just fetched (same swizzle as the TMA boxes) and to
          // the token's slot in the pool.
          const int rl = kv_len - 1 - j * SLAB, box = rl >> 4, r = rl & 15;
          const bool is_v = lane >= 8 * HALVES;
          const int cidx = lane - (is_v ? 8 * HALVES : 0);
          if (lane < 16 * HALVES) {
            const size_t row_off = (static_cast<size_t>(kvh) * D) * sizeof(T) + static_cast<size_t>(cidx) * 16;
            const size_t kv_row_bytes = static_cast<size_t>(a.kv_heads) * D * sizeof(T);
            const char* src = static_cast<const char*>(is_v ? a.new_v : a.new_k) + static_cast<size_t>(token) * kv_row_bytes + row_off;
            const uint4 val = __ldg(reinterpret_cast<const uint4*>(src));
            char* pool = static_cast<char*>(const_cast<void*>(is_v ? a.v_cache : a.k_cache));
            *reinterpret_cast<uint4*>(pool + static_cast<size_t>(__ldg(a.slots + token)) * kv_row_bytes + row_off) = val;
            unsigned char* dst = ring_ptr + slot * S::kStageBytes + (is_v ? S::kKBytes : 0) +
                                 (box * HALVES + (cidx >> 3)) * kBoxBytes + r * 128 + (((cidx & 7) ^ (r & 7)) << 4);
            *reinterpret_cast<uint4*>(dst) = val;
          }
          __syncwarp();
        }
      }
      if (rows_valid < SLAB) {
        // Slots past the end of the history hold whatever was there before (or were
        // never fetched): their scores are masked below, and their V rows are
        // cleared here so that 0 * garbage cannot produce a NaN.
        unsigned char* vptr = ring_ptr + slot * S::kStageBytes + S::kKBytes;
        const int nrows = SLAB - rows_valid;
        for (int i = lane; i < nrows * 8 * HALVES; i += 32) {
          const int row = rows_valid + i / (8 * HALVES);
          const int rem = i % (8 * HALVES);
          const int h = rem >> 3, ch = rem & 7;
          *reinterpret_cast<uint4*>(vptr + ((row >> 4) * HALVES + h) * kBoxBytes + (row & 15) * 128 + ch * 16) =
              make_uint4(0u, 0u, 0u, 0u);
        }
        __syncwarp();
      }

      if constexpr (F32) {
        // Scores: each lane half a row of K against the eight query rows, all from shared memory (16-byte reads:
        // the K rows swizzled, the query rows broadcast), two partial sums per head.  One slab of 8 KB costs a
        // warp about 600 issue slots, so twelve warps on an SM keep up with twice its share of HBM.
        const unsigned char* kp = ring_ptr + slot * S::kStageBytes;
        const unsigned char* vp = kp + S::kKBytes;
        float2 s2[8];
#pragma unroll
        for (int h = 0; h < 8; ++h) s2[h] = make_float2(0.f, 0.f);
#pragma unroll
        for (int b = 0; b < HALVES / 2; ++b)
#pragma unroll
          for (int ch = 0; ch < 8; ++ch) {
            const float4 kv = *reinterpret_cast<const float4*>(kp + (f_part * (HALVES / 2) + b) * kBoxBytes + f_key * 128 + ((ch ^ (f_key & 7)) << 4));
            const float* qd = f_q + f_part * (D / 2 + 4) + b * 32 + ch * 4;
#pragma unroll
            for (int h = 0; h < 8; ++h) {
              const float4 qv = *reinterpret_cast<const float4*>(qd + h * (D + 4));
              s2[h] = fma2(make_float2(kv.x, kv.y), make_float2(qv.x, qv.y), s2[h]);
              s2[h] = fma2(make_float2(kv.z, kv.w), make_float2(qv.z, qv.w), s2[h]);
            }
          }
        // the halves of the warp trade halves of the dims for halves of the heads
        float p[4], al[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float lo = s2[i].x + s2[i].y, hi = s2[4 + i].x + s2[4 + i].y;
          const float got = __shfl_xor_sync(0xffffffffu, f_part ? lo : hi, 16);
          const float sc = f_key < rows_valid ? ((f_part ? hi : lo) + got) * a.scale : -INFINITY;
          float mx = sc;
#pragma unroll
          for (int off = 1; off < 16; off <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
          const float mn = fmaxf(f_m[i], mx);            // finite: key 0 of a slab is valid
          al[i] = expf(f_m[i] - mn);
          p[i] = expf(sc - mn);
          f_l[i] = f_l[i] * al[i] + p[i];
          f_m[i] = mn;
        }
        // weights [key][head] and rescale factors over the K rows, which nothing reads any more
        float* sp = reinterpret_cast<float*>(ring_ptr + slot * S::kStageBytes);
        __syncwarp();
        *reinterpret_cast<float4*>(sp + f_key * 8 + f_part * 4) = make_float4(p[0], p[1], p[2], p[3]);
        if (f_key == 0) *reinterpret_cast<float4*>(sp + 128 + f_part * 4) = make_float4(al[0], al[1], al[2], al[3]);
        __syncwarp();
        {
          const float4 a0 = *reinterpret_cast<const float4*>(sp + 128), a1 = *reinterpret_cast<const float4*>(sp + 132);
          const float alpha[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
          for (int h = 0; h < 8; ++h)
#pragma unroll
            for (int x = 0; x < D / 64; ++x) { f_o[h][x].x *= alpha[h]; f_o[h][x].y *= alpha[h]; }
        }
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          float2 v[D / 64];
          if constexpr (D == 64) {
            v[0] = *reinterpret_cast<const float2*>(vp + f_part * kBoxBytes + k * 128 + ((((lane & 15) >> 1) ^ (k & 7)) << 4) + (lane & 1) * 8);
          } else {
            const float4 w = *reinterpret_cast<const float4*>(vp + (lane >> 3) * kBoxBytes + k * 128 + (((lane & 7) ^ (k & 7)) << 4));
            v[0] = make_float2(w.x, w.y);
            v[D / 64 - 1] = make_float2(w.z, w.w);
          }
          const float4 p0 = *reinterpret_cast<const float4*>(sp + k * 8), p1 = *reinterpret_cast<const float4*>(sp + k * 8 + 4);
          const float pk[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
#pragma unroll
          for (int h = 0; h < 8; ++h)
#pragma unroll
            for (int x = 0; x < D / 64; ++x) f_o[h][x] = fma2(make_float2(pk[h], pk[h]), v[x], f_o[h][x]);
        }
      } else {
      // S^T = K Q^T : MT m-tiles of 16 keys.
      float s[MT][NT][4];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) s[mt][nt][0] = s[mt][nt][1] = s[mt][nt][2] = s[mt][nt][3] = 0.f;
        const int row16 = ((mi & 1) << 3) + r8;
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
          const int chunk = 2 * ks + (mi >> 1);
          const uint32_t addr = kst + (mt * HALVES + (chunk >> 3)) * kBoxBytes + row16 * 128 + (((chunk & 7) ^ r8) << 4);
          uint32_t ka[4];
          ldmatrix_x4(addr, ka[0], ka[1], ka[2], ka[3]);
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) mma16816<T>(s[mt][nt], ka, qb[ks][nt][0], qb[ks][nt][1]);
        }
      }
      if (rows_valid < SLAB) {
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (16 * mt + g + 8 * (e >> 1) >= rows_valid) s[mt][nt][e] = -INFINITY;
      }
      // Online softmax, per head (thread holds heads 8nt+2c and 8nt+2c+1).
      uint32_t pb[MT][NT][2];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        float mx0 = fmaxf(s[0][nt][0], s[0][nt][2]);
        float mx1 = fmaxf(s[0][nt][1], s[0][nt][3]);
#pragma unroll
        for (int mt = 1; mt < MT; ++mt) {
          mx0 = fmaxf(mx0, fmaxf(s[mt][nt][0], s[mt][nt][2]));
          mx1 = fmaxf(mx1, fmaxf(s[mt][nt][1], s[mt][nt][3]));
        }
#pragma unroll
        for (int off = 4; off < 32; off <<= 1) {
          mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, off));
          mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, off));
        }
        const float mn0 = fmaxf(m_run[nt][0], mx0), mn1 = fmaxf(m_run[nt][1], mx1);
        const float al0 = exp2f((m_run[nt][0] - mn0) * sl2), al1 = exp2f((m_run[nt][1] - mn1) * sl2);
        m_run[nt][0] = mn0;
        m_run[nt][1] = mn1;
        const float ng0 = -mn0 * sl2, ng1 = -mn1 * sl2;
        float ps0 = 0.f, ps1 = 0.f;
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          const float p0 = exp2f(fmaf(s[mt][nt][0], sl2, ng0)), p1 = exp2f(fmaf(s[mt][nt][1], sl2, ng1));
          const float p2 = exp2f(fmaf(s[mt][nt][2], sl2, ng0)), p3 = exp2f(fmaf(s[mt][nt][3], sl2, ng1));
          ps0 += p0 + p2;
          ps1 += p1 + p3;
          // (key g | g+8 ; heads 2c, 2c+1)  ->  (head g ; keys 2c, 2c+1): the B operand of O^T += V^T P^T
          movmatrix_trans(pb[mt][nt][0], pack2<T>(p0, p1));
          movmatrix_trans(pb[mt][nt][1], pack2<T>(p2, p3));
        }
        l_run[nt][0] = l_run[nt][0] * al0 + ps0;
        l_run[nt][1] = l_run[nt][1] * al1 + ps1;
#pragma unroll
        for (int dm = 0; dm < KS; ++dm) {
          o[dm][nt][0] *= al0;
          o[dm][nt][1] *= al1;
          o[dm][nt][2] *= al0;
          o[dm][nt][3] *= al1;
        }
      }
      // O^T += V^T P^T : m-tiles of 16 dims, k = the slab's keys.
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        const int row16 = ((mi >> 1) << 3) + r8;
#pragma unroll
        for (int dm = 0; dm < KS; ++dm) {
          const int chunk = 2 * dm + (mi & 1);
          const uint32_t addr = vst + (mt * HALVES + (chunk >> 3)) * kBoxBytes + row16 * 128 + (((chunk & 7) ^ r8) << 4);
          uint32_t va[4];
          ldmatrix_x4_trans(addr, va[0], va[1], va[2], va[3]);
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) mma16816<T>(o[dm][nt], va, pb[mt][nt][0], pb[mt][nt][1]);
        }
      }
      }
      ++n_consumed;
    }
    if (!ok) {
      // The copies still on their way into this warp's ring are waited for (as long again, once each): the ring's
      // memory goes to another block when this one leaves.
      for (uint32_t i = n_consumed; i != n_issued; ++i) mbar_wait(bars + 8 * (i % NSTAGES), (i / NSTAGES) & 1u);
      if constexpr (!CLUSTER) break;   // (in a cluster the warp stays for the barriers; its give-up is on record)
    }

    while (more && n_issued - n_consumed < NSTAGES) more = issue_next();  // keep loads flowing through the finish

    // ------------------------------ finish the unit ------------------------------
    if constexpr (F32) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int off = 1; off < 16; off <<= 1) f_l[i] += __shfl_xor_sync(0xffffffffu, f_l[i], off);
      const int head0 = kvh * a.group, d0 = lane * (D / 32);
      if (part < 0) {
        float* out = reinterpret_cast<float*>(out_row<T>(a, a.out, token)) + static_cast<size_t>(head0) * D + d0;
#pragma unroll
        for (int h = 0; h < 8; ++h) {
          const float inv = 1.f / __shfl_sync(0xffffffffu, f_l[h & 3], (h >> 2) * 16);
          if (h < a.group)
#pragma unroll
            for (int x = 0; x < D / 64; ++x)
              *reinterpret_cast<float2*>(out + static_cast<size_t>(h) * D + 2 * x) = make_float2(f_o[h][x].x * inv, f_o[h][x].y * inv);
        }
      } else {
        __syncwarp();     // (cluster launches: the partial goes over the ring, which other lanes may still be reading)
        float* pacc = CLUSTER ? reinterpret_cast<float*>(ring_ptr) : a.part_acc + (static_cast<size_t>(part) * a.q_heads + head0) * D;
        float* pml = CLUSTER ? reinterpret_cast<float*>(ring_ptr) + 8 * D : a.part_ml + (static_cast<size_t>(part) * a.q_heads + head0) * 2;
#pragma unroll
        for (int h = 0; h < 8; ++h)
          if (h < a.group)
#pragma unroll
            for (int x = 0; x < D / 64; ++x) *reinterpret_cast<float2*>(pacc + static_cast<size_t>(h) * D + d0 + 2 * x) = f_o[h][x];
        if (f_key == 0)
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (4 * f_part + i < a.group) { pml[2 * (4 * f_part + i)] = f_m[i]; pml[2 * (4 * f_part + i) + 1] = f_l[i]; }
      }
    }
    if constexpr (!F32) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
      for (int off = 4; off < 32; off <<= 1) {
        l_run[nt][0] += __shfl_xor_sync(0xffffffffu, l_run[nt][0], off);
        l_run[nt][1] += __shfl_xor_sync(0xffffffffu, l_run[nt][1], off);
      }
    }
    const int head_base = kvh * a.group;
    if (TOK == 1 && part < 0) {
      T* out = out_row<T>(a, a.out, token) + static_cast<size_t>(head_base) * D;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const int h0 = 8 * nt + 2 * c;
        const float i0 = 1.f / l_run[nt][0], i1 = 1.f / l_run[nt][1];
#pragma unroll
        for (int dm = 0; dm < KS; ++dm) {
          const int d = 16 * dm + g;
          if (h0 < a.group) {
            out[static_cast<size_t>(h0) * D + d] = Elem<T>::from_f32(o[dm][nt][0] * i0);
            out[static_cast<size_t>(h0) * D + d + 8] = Elem<T>::from_f32(o[dm][nt][2] * i0);
          }
          if (h0 + 1 < a.group) {
            out[static_cast<size_t>(h0 + 1) * D + d] = Elem<T>::from_f32(o[dm][nt][1] * i1);
            out[static_cast<size_t>(h0 + 1) * D + d + 8] = Elem<T>::from_f32(o[dm][nt][3] * i1);
          }
        }
      }
    } else {
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const int ti = nt / NTG;
        if (ti >= n_tok) continue;
        // the partial: to the workspace, or (cluster launches) to the start of this warp's own ring,
        // which holds no copy in flight any more -- [8 NT heads][D] sums, then (maximum, sum) per head
        float* pacc = CLUSTER ? reinterpret_cast<float*>(ring_ptr)
                              : a.part_acc + (static_cast<size_t>(parts[ti]) * a.q_heads + head_base) * D;
        float* pml = CLUSTER ? reinterpret_cast<float*>(ring_ptr) + 8 * NT * D
                             : a.part_ml + (static_cast<size_t>(parts[ti]) * a.q_heads + head_base) * 2;
        const int h0 = 8 * (nt % NTG) + 2 * c;
#pragma unroll
        for (int dm = 0; dm < KS; ++dm) {
          const int d = 16 * dm + g;
          if (h0 < a.group) {
            pacc[static_cast<size_t>(h0) * D + d] = o[dm][nt][0];
            pacc[static_cast<size_t>(h0) * D + d + 8] = o[dm][nt][2];
          }
          if (h0 + 1 < a.group) {
            pacc[static_cast<size_t>(h0 + 1) * D + d] = o[dm][nt][1];
            pacc[static_cast<size_t>(h0 + 1) * D + d + 8] = o[dm][nt][3];
          }
        }
        if (g == 0) {
          if (h0 < a.group) { pml[2 * h0] = m_run[nt][0] * sl2; pml[2 * h0 + 1] = l_run[nt][0]; }
          if (h0 + 1 < a.group) { pml[2 * h0 + 2] = m_run[nt][1] * sl2; pml[2 * h0 + 3] = l_run[nt][1]; }
        }
      }
    }
    }
  }
  if constexpr (!CLUSTER && !FUSED_APPEND) {
    // This launch's completion has to imply the previous one's: one block stays for it.  (All of them waiting
    // here kept the blocks that had found no room yet from starting before the previous launch's end.)
    if (a.wait_last && blockIdx.x == 0) pdl_wait();
  }
  if constexpr (CLUSTER) {
    if (c_nsplits > 1) {               // the same for every thread of the cluster
      if (!waited) pdl_wait();         // warps without a range write output rows too
      asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");   // every block's landing barrier is armed
      const uint32_t land0 = ring0 + WARPS * (S::kWarpBytes + S::kQBytes);    // landing area: behind the rings
      const int ranges_max = WARPS * static_cast<int>(c_size);
      if (c_len > 0) {
        // send this warp's partial, head by head, to the heads' owners: D / 4 quads of sums and one with
        // (maximum, sum) per head, read back from where the unit's finish left them
        __syncwarp();
        const float* pacc = reinterpret_cast<const float*>(ring_ptr);
        const float* pml = pacc + 8 * NT * D;
        for (int i = lane; i < a.group * (D / 4 + 1); i += 32) {
          const int h = i / (D / 4 + 1), k = i - h * (D / 4 + 1);
          const uint32_t owner = static_cast<uint32_t>(h) % c_size, j = static_cast<uint32_t>(h) / c_size;
          float4 v;
          if (k < D / 4) {
            v = *reinterpret_cast<const float4*>(pacc + h * D + 4 * k);
          } else {
            const float2 ml = *reinterpret_cast<const float2*>(pml + 2 * h);
            v = make_float4(ml.x, ml.y, 0.f, 0.f);
          }
          const uint32_t dst = land0 + (j * ranges_max + c_split) * kClusterRecord + 16 * k;
          cluster_push4(cluster_map(dst, owner), v, cluster_map(smem_u32(&land_bar), owner));
        }
      }
      // this block's heads: wait for all their records, fold them, write the rows
      if (!mbar_wait(smem_u32(&land_bar), 0u)) {
        if (threadIdx.x == 0) report_give_up(a, kErrConsumerWait);
      }
      const int owned = (a.group - static_cast<int>(c_rank) + static_cast<int>(c_size) - 1) / static_cast<int>(c_size);
      const unsigned char* land_ptr = smem_raw + (land0 - smem_u32(smem_raw));
      for (int e = threadIdx.x; e < owned * (D / 2); e += WARPS * 32) {     // one pair of dims per thread
        const int j = e / (D / 2), d = 2 * (e - j * (D / 2));
        const int h = j * static_cast<int>(c_size) + static_cast<int>(c_rank);
        const unsigned char* rec0 = land_ptr + static_cast<size_t>(j) * ranges_max * kClusterRecord;
        float m_run = -INFINITY;
#pragma unroll 4
        for (int sp = 0; sp < c_nsplits; ++sp) m_run = fmaxf(m_run, *reinterpret_cast<const float*>(rec0 + sp * kClusterRecord + 4 * D));
        float l_run = 0.f, acc0 = 0.f, acc1 = 0.f;
#pragma unroll 4
        for (int sp = 0; sp < c_nsplits; ++sp) {
          const unsigned char* rec = rec0 + sp * kClusterRecord;
          const float2 ml = *reinterpret_cast<const float2*>(rec + 4 * D);
          const float f = (ml.x == -INFINITY) ? 0.f : softmax_exp<!F32>(ml.x - m_run);
          const float2 v = *reinterpret_cast<const float2*>(rec + 4 * d);
          l_run += f * ml.y;
          acc0 += f * v.x;
          acc1 += f * v.y;
        }
        const float inv = 1.f / l_run;
        T* o = out_row<T>(a, a.out, c_token) + static_cast<size_t>(c_kvh * a.group + h) * D + d;
        if constexpr (F32) *reinterpret_cast<float2*>(o) = make_float2(acc0 * inv, acc1 * inv);
        else *reinterpret_cast<uint32_t*>(o) = pack2<T>(acc0 * inv, acc1 * inv);
      }
    }
  }
}

}  // namespace pkv
