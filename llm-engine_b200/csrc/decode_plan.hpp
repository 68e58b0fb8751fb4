// Split-K work list for paged decode attention: layout of the caller's workspace
// and the rule that picks the chunk size.  Shared by the host planner, the device
// planner kernel and the attention kernels, so all three agree by construction.
//
// A decode step is a ragged batch: token t attends L_t = token_pos[t] + 1 keys and
// L_t can differ by 64x inside one batch.  One thread block per (token, kv head)
// would leave the GPU waiting for the longest sequence, so each token's key range
// is cut; a work item is (token, first key, key count).  Tokens that stay whole write
// their output directly; the others write one partial (running max, denominator,
// unnormalised accumulator) per item, and a second kernel merges them.
//
// Two ways to cut (ShareRule below): steps with enough keys are laid end to end and cut
// into equal SHARES, one per resident warp and kv head, so that every warp reads the same
// number of keys and a token has a partial per warp that touches it and no more; small
// steps are cut token by token into chunks.
//
// Workspace layout (every region 256-byte aligned):
//   header | tok_split[n_tokens] | counters[n_tokens*kv_heads] | items[cap_items]
//          | part_ml[cap_parts*q_heads*2] | part_acc[cap_parts*q_heads*head_dim]
// The first four regions up to items[n_items] (and, behind the items of a plan with shares,
// the first item of every share) form the "plan image" that the host planner uploads in one copy.
#pragma once

#include <cstddef>
#include <cstdint>

#if defined(__CUDACC__)
#define PKV_HD __host__ __device__
#else
#define PKV_HD
#endif

namespace pkv {

constexpr int kPlanMagic = 0x706b7631;  // "pkv1"
constexpr int kNumChunkCandidates = 9;  // 64, 128, ..., 16384 keys
constexpr int kMinChunk = 64;

struct PlanHeader {
  int magic;
  int n_items;
  int chunk;  // 0 = tokens are not split
  int n_tokens;
  int n_parts;
  int kv_heads;
  int n_shares;  // 0: units are dealt one by one; otherwise int first_item[n_shares + 1] follows the items
  int pad;
};

struct WorkItem {
  int token;
  int kv_begin;
  int kv_len;
  int part;  // partial slot to write, or -1 to write the final output directly
};

// A unit of the shared-prefix planner: up to four tokens whose sequences have the same blocks
// over keys [kv_begin, kv_begin + kv_len); each token's partial goes to its own slot.  Stored
// behind the ordinary items in the same workspace region, three 16-byte slots each.
struct SharedItem {
  int kv_begin, kv_len, n_tok, pad;
  int token[4];
  int part[4];
};
static_assert(sizeof(SharedItem) == 3 * sizeof(WorkItem), "three item slots");
constexpr int kSharedTokens = 4;

struct TokSplit {
  int part_base;  // first partial slot of this token (valid when nsplits > 1)
  int nsplits;
};

struct WsLayout {
  size_t off_tok, off_cnt, off_items, off_ml, off_acc, total;
  int cap_extra;  // items beyond one per token that fit
  int cap_items, cap_parts;
};

PKV_HD inline size_t align256(size_t x) { return (x + 255) & ~static_cast<size_t>(255); }

// Layout for a workspace that admits `extra` work items beyond one per token
// (and therefore at most 2*extra partial slots: a token that is split at all
// contributes at least two items for one item of excess).
PKV_HD inline WsLayout ws_layout(int n_tokens, int q_heads, int kv_heads, int head_dim, int extra) {
  WsLayout w;
  w.cap_extra = extra;
  w.cap_items = n_tokens + extra;
  w.cap_parts = 2 * extra;
  size_t o = align256(sizeof(PlanHeader));
  w.off_tok = o;
  o = align256(o + sizeof(TokSplit) * static_cast<size_t>(n_tokens));
  w.off_cnt = o;
  o = align256(o + sizeof(int) * static_cast<size_t>(n_tokens) * kv_heads);
  w.off_items = o;
  o = align256(o + sizeof(WorkItem) * static_cast<size_t>(w.cap_items));
  w.off_ml = o;
  o = align256(o + sizeof(float) * 2 * static_cast<size_t>(w.cap_parts) * q_heads);
  w.off_acc = o;
  o = align256(o + sizeof(float) * static_cast<size_t>(w.cap_parts) * q_heads * head_dim);
  w.total = o;
  return w;
}

// Largest `extra` whose layout fits in `bytes`, or -1 if not even extra = 0 fits.
inline int ws_extra_for_bytes(int n_tokens, int q_heads, int kv_heads, int head_dim, size_t bytes, int max_extra) {
  if (ws_layout(n_tokens, q_heads, kv_heads, head_dim, 0).total > bytes) return -1;
  int lo = 0, hi = max_extra;
  while (lo < hi) {
    const int mid = lo + (hi - lo + 1) / 2;
    if (ws_layout(n_tokens, q_heads, kv_heads, head_dim, mid).total <= bytes) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// ---- shares -----------------------------------------------------------------------
// The tokens' histories, each rounded up to whole slabs, are laid end to end; share j is the
// stretch [j * per, (j + 1) * per).  A token is cut at every multiple of `per` that lies more
// than a slab inside it on both sides, and an item belongs to the share its first key falls
// into, give or take that slab: shares stay within a slab of `per`, no piece of a cut token is
// a lone slab, and every share but possibly the last begins with exactly one item.
//
// Cutting every token into chunks of its own (256 keys and up, dealt round-robin) gave a step of
// 256 sequences x 128-8,192 keys on 4 kv heads 1,440 items a kv head for 444 warps: a third more
// or less work on some warps and 1,100 partials, where shares give each warp the same 1,145 keys
// and 650 partials.
constexpr int kShareSlab = 32;
// Below this many keys a share the tokens are cut one by one into chunks instead (chunk_rule): equal shares would cut
// short tokens that need no merge at all when left whole.
constexpr int kMinShareKeys = 128;
// A plan listed longest first does better with chunks up to this many keys a share, too, if its tokens are mostly
// shorter than two shares (600 tokens of 60-700 keys, us a layer: 2 kv heads, 180 keys a share, shares 26.5, chunks 25.8;
// but 8 of 3,000 at 8 kv heads, 162 keys a share, 27.2 and 28.9).
constexpr int kMinSortedShareKeys = 192;
// Chunks go down to this length when there are so few keys a share that the longest units decide: four dependent slabs
// a warp become two.  Only in steps planned on the device that have no prefill chunk, whose kernel the decode units
// hide behind, and no token of so many chunks that their merge outweighs the shorter units; small host-planned steps take
// the cluster form.  Engine decode steps, us a layer with 128- and 64-key chunks: 1 sequence of 333 keys 11.7, 10.2; 6 of 100-900
// (4 kv heads) 12.4, 11.0; 40 of 50-1,000 14.7, 13.3 (15 keys a share); 60 of 60-300 16.3, 15.1 (23); 80 of 60-300 16.7, 15.9
// (31); and without a caller's plan 1 of 8,000 16.8, 20.6, 8 of 3,000 13.4, 15.5.
constexpr int kFineChunk = 64;
constexpr int kFineShareKeys = 36;
constexpr int kFineMaxKeys = 2048;

PKV_HD inline int share_padded(int len) { return (len + kShareSlab - 1) & ~(kShareSlab - 1); }

struct ShareCut {
  long long first;   // first cut, in the laid-out coordinate (valid when n > 0)
  int n;             // cuts: the token has n + 1 items
};
// Cuts of a token that begins at `begin` and is `padded` keys long (> 0).
PKV_HD inline ShareCut share_cuts(long long begin, int padded, int per) {
  ShareCut c;
  c.first = ((begin + kShareSlab) / per + 1) * per;
  const long long end = begin + padded - kShareSlab;    // cuts lie strictly below
  c.n = end > c.first ? static_cast<int>((end - 1 - c.first) / per) + 1 : 0;
  return c;
}
// Share of the item that begins at `item_begin` (a last token of one slab would otherwise open a share of its own).
PKV_HD inline int share_of(long long item_begin, int per, int n_shares) {
  const long long s = (item_begin + kShareSlab) / per;
  return static_cast<int>(s < n_shares ? s : n_shares - 1);
}

struct ShareRule {
  int per;        // keys per share (a multiple of the slab), or 0: cut token by token
  int n_shares;
  int chunk;      // per == 0: keys per chunk, 0 = tokens are not cut
};
// What a plan is made for and may use.
struct PlanLimits {
  int max_shares;    // warps per kv head, as far as the workspace has room for their partials
  int max_extra;     // items beyond one per token
  int kv_heads;
  int wave_units;    // units that keep the GPU busy
  int forced_chunk;  // 0: the rules below
  int shares;        // whether shares are for the kernel of this geometry: not for the SIMT kernel, which gives an item a
                     // block and wants long ones first (200 tokens of 100-2,000 keys at head_dim 96: 114 us a layer in
                     // shares, 101 in chunks)
  int sorted;        // whether chunks are listed longest first (the host's planner)
};
// Keys per chunk when tokens are cut one by one: the smallest of 256, 512, ... that the workspace has room for, 128
// where that leaves fewer units than the GPU has workers, 0 when nothing fits.  A token of L keys has at most L / chunk
// items beyond its first, so the step's total bounds their sum.
PKV_HD inline int chunk_rule(long long total, int n_tokens, const PlanLimits& lim) {
  int log2 = 8;
  while (log2 <= 14 && (total >> log2) > lim.max_extra) ++log2;
  if (log2 > 14) return 0;
  const long long items = (total >> 8) + n_tokens / 2;      // of 256 keys, about
  if (log2 == 8 && (items > n_tokens ? items : n_tokens) * lim.kv_heads < lim.wave_units && (total >> 7) <= lim.max_extra) log2 = 7;
  return 1 << log2;
}
// The rule for plans in token order.  slabs: of the whole step; longest: keys of its longest token; max_shares: as below;
// fine: see kFineChunk.  A chunk of 128 or 64 keys makes fewer extra items than there may be shares.
template <typename Int>
PKV_HD inline ShareRule ordered_share_rule(Int slabs, int longest, int max_shares, bool fine) {
  ShareRule r{0, 0, 0};
  if (max_shares <= 0) return r;
  const Int most = max_shares;
  if (slabs < most * (kMinShareKeys / kShareSlab)) {
    r.chunk = fine && longest > 128 && longest <= kFineMaxKeys && slabs * kShareSlab < most * kFineShareKeys ? kFineChunk : kMinShareKeys;
    return r;
  }
  // many tokens, all short: whole (a plan that is sorted leaves more of them whole, see share_rule)
  if (longest <= 128) { r.chunk = 256; return r; }
  const Int per = (slabs + most - 1) / most;
  if (per > 0x40000000 / kShareSlab) return r;
  r.per = static_cast<int>(per) * kShareSlab;
  r.n_shares = static_cast<int>((slabs + per - 1) / per);
  return r;
}
// total: padded keys of the step.
PKV_HD inline ShareRule share_rule(long long total, int longest, int n_tokens, const PlanLimits& lim, bool fine) {
  ShareRule r{0, 0, 0};
  if (lim.max_shares <= 0) return r;
  if (lim.forced_chunk > 0 && total / lim.forced_chunk <= lim.max_extra) { r.chunk = lim.forced_chunk; return r; }
  const bool few = total < static_cast<long long>(lim.max_shares) * kMinShareKeys;
  if (!few && !lim.shares) { r.chunk = chunk_rule(total, n_tokens, lim); return r; }
  r = ordered_share_rule<long long>(total / kShareSlab, longest, lim.max_shares, fine);
  if (lim.sorted) {
    const int chunk = chunk_rule(total, n_tokens, lim);
    // Enough tokens to fill the GPU, none of them cut: shares would add the merge for nothing (1,000 tokens of 20 to 200
    // keys, us a layer: 4 kv heads 31.0 in shares, 26.3 whole; 2 kv heads 19.0, 14.6.  In token order they are balanced
    // better by shares: 34.3 against 36.2).
    if ((few && longest > 128) || (!few && chunk == 256 && longest <= 256) ||
        (r.per > 0 && r.per <= kMinSortedShareKeys && total < 2ll * r.per * n_tokens)) r = ShareRule{0, 0, chunk};
  }
  return r;
}
// Shares a workspace with room for `extra` items beyond one per token takes: the items, their
// partials and the table behind the items.
PKV_HD inline int max_shares_for(int extra, int workers_per_kv_head) {
  const int fit = (extra - 2) / 5 * 4;
  return fit < workers_per_kv_head ? (fit > 0 ? fit : 0) : workers_per_kv_head;
}

// ---- steps planned inside the kernels ------------------------------------------------
// Steps of up to this many tokens whose caller brings no plan need no planner launch: every block of the decode
// kernel finds the cuts for itself (14 bytes of shared memory a token, which is what three blocks on an SM
// leave), and in mixed steps every block of the prefill kernel the long runs.
constexpr int kInlineTokens = 704;
constexpr int kInlineRuns = 256;
struct InlineRuns {
  const int* token_pos;
  const int* token_seq;
  const int* table_offset;
  int min_run;
};

// Chunk rule of the shared-prefix planner.  items_at[j] = sum over tokens of ceil(L_t / (64 << j)).
//   1. take the smallest chunk >= 256 keys whose item count stays within the
//      budget (one item per token plus `extra_budget`): the most parallelism the
//      workspace and the target grid allow, without paying a partial per 16 KB;
//   2. if that still leaves fewer units than the GPU has workers (warps), go down to
//      128 keys if the budget allows (64-key units were measured slower: the fixed
//      cost per unit outweighs the extra parallelism).
// Returns 0 when no candidate fits (tokens are then processed unsplit).
PKV_HD inline int choose_chunk(const long long* items_at, int n_tokens, int kv_heads, long long extra_budget,
                               int wave_ctas, int forced_chunk) {
  if (forced_chunk > 0) {
    for (int j = 0; j < kNumChunkCandidates; ++j)
      if ((kMinChunk << j) == forced_chunk && items_at[j] - n_tokens <= extra_budget) return forced_chunk;
  }
  int best = -1;
  for (int j = 2; j < kNumChunkCandidates; ++j) {
    if (items_at[j] - n_tokens <= extra_budget) { best = j; break; }
  }
  if (best < 0) return 0;
  if (best == 2 && items_at[best] * kv_heads < wave_ctas && items_at[1] - n_tokens <= extra_budget) best = 1;
  return kMinChunk << best;
}

}  // namespace pkv
