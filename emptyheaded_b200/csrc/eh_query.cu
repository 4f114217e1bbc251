// Generic-join COUNT executors for the named plans.
//
// Reference loop nest (triangle, order [a,b,c]; EHGenerator.scala:273-480,
// TrieBuilder.cpp:242-274, ParTrieBuilder::par_foreach_aggregate
// TrieBuilder.hpp:152-157):
//     for a in head ∩ head (parallel, par::for_range chunks):
//       for b in N(a) ∩ head:
//         count += |N(b) ∩ N(a)|          (ops::set_intersect, set.hpp:9-167)
// The same pairwise intersections are scheduled here grouped by b: N(b) is
// staged once in shared memory in its stored layout (uint -> sorted list,
// range bitset -> words, block bitset -> ids + words) and every row a->b
// streams the part of N(a) that can still meet N(b) (the reverse level of
// the trie, built with it).  The sum is unchanged: it is the same set of
// (a,b) intersections.  Work items are (b, range of rows a->b) chunks of
// about `chunk_pairs` probes, pulled by warps of a persistent kernel from
// an atomic queue, heaviest b first.
#include <algorithm>
#include <cstring>

#include "eh_internal.cuh"

namespace eh {

// Register budget of the intersection kernels, set by their launch bounds
// (threads per block, optional blocks per SM); the block size knob is
// capped to match.
#ifndef EH_TRI_MAX_THREADS
#define EH_TRI_MAX_THREADS 512
#endif
#ifdef EH_TRI_MIN_BLOCKS
#define EH_TRI_LAUNCH_BOUNDS __launch_bounds__(EH_TRI_MAX_THREADS, EH_TRI_MIN_BLOCKS)
#else
#define EH_TRI_LAUNCH_BOUNDS __launch_bounds__(EH_TRI_MAX_THREADS)
#endif
constexpr int kMaxWarps = EH_TRI_MAX_THREADS / 32;  // per block
constexpr int kDefaultWarps = kMaxWarps < 8 ? kMaxWarps : 8;
constexpr uint32_t kDefaultLongRow = 48;  // rows with at least this many candidates run warp-wide
#ifndef EH_LONG_UNROLL
#define EH_LONG_UNROLL 4
#endif
constexpr int kLongUnroll = EH_LONG_UNROLL;  // independent candidate loads per lane per trip
#ifndef EH_SHORT_UNROLL
#define EH_SHORT_UNROLL 4
#endif
constexpr int kShortUnroll = EH_SHORT_UNROLL;  // flattened (row, element) pairs per lane per trip
#ifndef EH_WORD_UNROLL
#define EH_WORD_UNROLL 1
#endif
constexpr int kWordUnroll = EH_WORD_UNROLL;  // flattened (row, word) pairs per lane per trip
#ifndef EH_LONG_WORD_UNROLL
#define EH_LONG_WORD_UNROLL 1
#endif
constexpr int kLongWordUnroll = EH_LONG_WORD_UNROLL;  // 16-byte N(a) loads per lane per trip of a long word row
#ifndef EH_WORD_ROW_NUM
#define EH_WORD_ROW_NUM 5
#endif
#ifndef EH_WORD_ROW_DEN
#define EH_WORD_ROW_DEN 4
#endif
// a row runs word by word when words * num < candidates * den: a word costs
// about 1.25 candidate probes (measured on B200 at R-MAT-22: 5/4 against 1/1
// 8.34 vs 8.46 ms with the per-set best layouts, 9.87 vs 9.91 with the rule)
constexpr uint32_t kWordRowNum = EH_WORD_ROW_NUM, kWordRowDen = EH_WORD_ROW_DEN;
#ifndef EH_LONG_WORDS
#define EH_LONG_WORDS 32
#endif
constexpr int kLongWords = EH_LONG_WORDS;  // word rows with at least this many words run warp-wide
// an item of at most this many rows and candidates keeps a uint N(b) as a list:
// searching it for so few beats building a bitmap (kernel ms, R-MAT-22 6.93 ->
// 6.85, symmetric Chung-Lu 2^21 2.52 -> 2.21, ER-16K 0.0225 -> 0.0205; at 32 rows
// R-MAT-22 6.96; without the bound on candidates a star of 2^16 leaves, whose rows
// hold 32 K of them, took 4.9 ms instead of 2.4)
constexpr uint32_t kListRows = 16;
constexpr uint64_t kListCandidates = 2048;
#ifndef EH_FLAT_CLIQUE
#define EH_FLAT_CLIQUE 48
#endif
constexpr uint32_t kFlatClique = EH_FLAT_CLIQUE;  // 4-clique: S up to this size has its pairs flattened
// Defaults measured on B200 at R-MAT-22 (5 KB of staging per warp leaves
// room for 32 resident warps; 1024 words 7.18 ms against 7.06); the
// autotuner (emptyheaded_b200/autotune.py) re-picks them per trie.
constexpr int kDefaultSmemWords = 1280;  // per warp
constexpr int kDefaultChunk = 32768;     // where it is not derived from the work (noalloc); 4-clique and annotation without masks: at most
constexpr uint64_t kMaxChunk = 131072;   // larger items amortise staging: 7.03 ms against 7.18 at 32768
constexpr uint64_t kMinChunk = 4096;  // the smallest item the planner cuts by itself
constexpr uint32_t kShareWarps = 148 * 32;  // resident warps of a B200 at the default schedule

struct RevView {
  const uint64_t* rev_off;
  const uint32_t* rev_lo;
  const uint32_t* rev_hi;
  const uint32_t* rev_src;
  const uint64_t* rev_wpre;
  int dir;
};

struct Item {  // 16 bytes
  uint32_t hb, kb, ke, g;
};

struct ExecParams {
  int warps;
  int smem_words;
  uint32_t chunk;
  uint32_t shard_index, shard_count;
  uint32_t long_row;
  uint32_t s_cap;  // 4-clique: S buffers in global memory of this many words per warp (0: in shared memory)
  bool smem_given; // the caller chose smem_words
  bool chunk_given;  // the caller chose chunk
  bool no_block_items;  // stage every N(b) per warp (no block items)
  bool masks = true;      // hit masks may be made
  bool* held = nullptr;   // set once they are
};

static ExecParams exec_params(const eh_exec_config* cfg) {
  ExecParams p;
  p.warps = (cfg && cfg->warps_per_block > 0) ? cfg->warps_per_block : kDefaultWarps;
  p.smem_words = (cfg && cfg->smem_words > 0) ? cfg->smem_words : kDefaultSmemWords;
  p.chunk_given = cfg && cfg->chunk_pairs > 0;
  p.chunk = p.chunk_given ? (uint32_t)cfg->chunk_pairs : (uint32_t)kDefaultChunk;
  p.long_row = (cfg && cfg->long_row > 0) ? (uint32_t)cfg->long_row : kDefaultLongRow;
  p.shard_count = (cfg && cfg->shard_count > 1) ? (uint32_t)cfg->shard_count : 1u;
  p.shard_index = (cfg && cfg->shard_count > 1) ? (uint32_t)cfg->shard_index : 0u;
  EH_REQUIRE(p.shard_index < p.shard_count, EH_ERR_INVALID, "shard_index must be below shard_count");
  p.s_cap = 0;
  p.smem_given = cfg && cfg->smem_words > 0;
  p.no_block_items = cfg && cfg->no_block_items;
  p.warps = std::max(1, std::min(p.warps, kMaxWarps));
  p.smem_words = std::max(64, std::min(p.smem_words, 16384)) & ~1;
  return p;
}

// ---------------------------------------------------------------- planning
// items per head entry b: ceil(work(b) / chunk)
__global__ void plan_count_kernel(RevView r, uint32_t nh, uint32_t chunk, uint32_t* __restrict__ nitems) {
  for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < nh; b += gridDim.x * blockDim.x) {
    const uint64_t w = r.rev_wpre[r.rev_off[b + 1]] - r.rev_wpre[r.rev_off[b]];
    nitems[b] = (uint32_t)((w + chunk - 1) / chunk);
  }
}
// item i of b covers the rows whose work prefix falls in [i, i+1) * W/n;
// items are written in reverse head order so the queue starts at the
// largest-degree b (ids are degree-ordered) and small items come last.
// first row k in [lo, hi) with wpre[k] >= target (hi if none)
__device__ __forceinline__ uint64_t first_row_at(const uint64_t* __restrict__ wpre, uint64_t lo, uint64_t hi,
                                                 uint64_t target) {
  while (lo < hi) {
    const uint64_t mid = (lo + hi) >> 1;
    if (wpre[mid] < target) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// One thread per item: item q belongs to the last head entry b with
// ipos[b] <= q (ipos is the exclusive scan of the items per entry, so entries
// without items share the next entry's offset and are never found), is item
// i = q - ipos[b] of b, and covers the rows from the first one at target i to
// the first one at target i + 1 -- two independent searches over b's rows.
// The work prefix is non-decreasing, so these are the bounds a serial cut of
// b's items one after the other finds, at any number of items per entry.
__global__ void plan_fill_scratch_kernel(RevView r, uint32_t nh, const uint32_t* __restrict__ nitems,
                                 const uint32_t* __restrict__ ipos, uint32_t total, uint32_t g,
                                 Item* __restrict__ items) {
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < total; q += gridDim.x * blockDim.x) {
    uint32_t lo = 0, hi = nh;  // first entry with ipos > q
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (ipos[mid] <= q) lo = mid + 1; else hi = mid;
    }
    const uint32_t b = lo - 1;  // q < total = ipos[nh-1] + nitems[nh-1], so lo >= 1
    const uint32_t i = q - ipos[b], n = nitems[b];
    const uint64_t k0 = r.rev_off[b], k1 = r.rev_off[b + 1];
    const uint64_t w0 = r.rev_wpre[k0], W = r.rev_wpre[k1] - w0;
    const uint64_t kb = i ? first_row_at(r.rev_wpre, k0, k1, w0 + (W * i) / n) : k0;
    const uint64_t ke = i + 1 < n ? first_row_at(r.rev_wpre, kb, k1, w0 + (W * (i + 1)) / n) : k1;
    items[total - 1 - q] = Item{b, (uint32_t)kb, (uint32_t)ke, g};
  }
}


// u32 words a compressed staging (P_ZBITS, below) of a W-word range bitset
// with len elements takes at most: a (presence mask, rank) pair per 32 words
// and at most min(len, W) non-zero 64-bit words
__host__ __device__ __forceinline__ uint32_t zbits_words(uint32_t W, uint32_t len) {
  const uint32_t groups = (W + 31) / 32;
  return 2 * groups + 2 * (len < W ? len : W);
}

// The part of N(b) the plans stage.  On a symmetric relation every row a->b
// runs with a < b and only candidates above b, so only N(b)'s elements above b
// can match: t.up[b] is the first of them, found once at build.  With ids in
// degree order that part is short even for a hub (Chung-Lu 2^21: sets of up to
// 630,714 elements, a few hundred of them above their own id), so it is staged in
// shared memory where the whole set had to be searched in global memory
// (lollipop there 36.6 -> 11.8 ms, barbell on 2^16 nodes 2.5 -> 1.5 ms).  Other relations stage the whole set.  No
// row of the reverse level has a b without such elements.
struct StagedRange {
  uint64_t s0;   // first element in vals
  uint32_t len;
};
__device__ __forceinline__ StagedRange staged_range(const TrieView& t, uint32_t b) {
  const uint64_t s0 = t.up ? (uint64_t)__ldg(t.up + b) : t.off[b];
  return StagedRange{s0, (uint32_t)(t.off[b + 1] - s0)};
}
// the same part of a range bitset: from the word of its first element on
__device__ __forceinline__ SetAux staged_bits(const TrieView& t, uint32_t b, const StagedRange& sr) {
  SetAux a = t.aux[b];
  if (t.up && sr.len) {
    const uint32_t skip = (__ldg(t.vals + sr.s0) >> 6) - a.start;
    a.off += skip;
    a.start += skip;
    a.n -= skip;
  }
  return a;
}

// Work of head entry b is staged in one of two classes: per warp (N(b)
// fits a warp's shared region, or must be probed in global memory) or per
// block (N(b) needs more than a warp's region but fits the block's: every
// warp of the block works on the rows of one staged N(b)).  A block item
// holds `warps` times a warp item's work.
__device__ __forceinline__ uint32_t staged_words(const TrieView& t, uint32_t b, uint32_t warp_words) {
  const uint8_t l = t.layout[b];
  const StagedRange sr = staged_range(t, b);
  if (l == EH_LAYOUT_RANGE_BITSET) {
    const uint32_t words = staged_bits(t, b, sr).n;
    const uint32_t raw = 2u * words;
    if (raw <= warp_words) return raw;
    const uint32_t z = zbits_words(words, sr.len);
    return z <= warp_words ? z : raw;  // compressed in a warp, or raw across a block
  }
  if (l == EH_LAYOUT_UINTEGER) return sr.len;
  return 0xffffffffu;  // block bitsets are probed in global memory
}

// A block item keeps every warp of the block on one staged N(b); a b with
// little work would leave most of them idle, so only a b with at least this
// many probes becomes block items (about 32 batches of 32 rows at R-MAT's
// row lengths); the others stay warp items probing N(b) in global memory.
#ifndef EH_MIN_BLOCK_WORK
#define EH_MIN_BLOCK_WORK (1ull << 17)
#endif
constexpr uint64_t kMinBlockWork = EH_MIN_BLOCK_WORK;

struct PlanShape {
  uint32_t chunk;        // probes per warp item
  const float* pred;     // predicted cycles of each head entry's work (learned layouts), or null
  double unit;           // predicted cycles per warp item
  uint32_t warp_words;   // staging capacity of a warp (u32 words)
  uint32_t block_words;  // staging capacity of a block; 0: no block items
  uint32_t warps;        // warps per block
  uint32_t merge;        // 1: neighbouring entries with little work share an item
};

// Cost of a row beside its candidates, in candidates: a row of one candidate
// takes its share of a batch's loads, scans and owner searches.  Without it an
// item of a hub's one-candidate rows held 32,768 rows and ran alone at the end
// (hit masks of Chung-Lu 2^20: SMs busy 56% of the kernel's time).
#ifndef EH_ROW_COST
#define EH_ROW_COST 8
#endif
constexpr uint32_t kRowCost = EH_ROW_COST;

// the first row k in [k0, k1) before which rows and candidates cost at least
// `target` (k1 if none)
__device__ __forceinline__ uint64_t row_at_cost(const uint64_t* __restrict__ wpre, uint64_t k0, uint64_t k1,
                                                uint64_t w0, uint64_t target) {
  uint64_t lo = k0, hi = k1;
  while (lo < hi) {
    const uint64_t mid = (lo + hi) >> 1;
    if (wpre[mid] - w0 + kRowCost * (mid - k0) < target) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// What a launch reads and writes beside the tries: the queues, the numbers of
// items the planner made, the results.  One copy from pinned host memory sets
// it up together with the views, one copy brings it back.
// The queue heads have a 128-byte line of their own: every item pulled is an
// atomic on it, and the warps read the rest (one line for all: triangle
// R-MAT-22 8.61 -> 8.89 ms).
struct Control {
  unsigned int queue[2];   // warp items, block items (or second-pass units)
  unsigned int pad0[30];
  unsigned int items[2];   // warp items, block items
  unsigned int pad1[30];
  unsigned long long spare[2];  // a total nobody reads; the planner's total of a trie
  // followed by unsigned long long total[n], then the views
};

// The plan of a trie, in three launches and without the host: how many items
// each head entry gives (and the sums over tiles of kPlanTile entries), where
// they go, and the items, one thread each.  The intersection kernel reads the
// number of items from the control block.  Items lie in reverse head order
// (ids are degree-ordered), so the queue starts at the heaviest b and small
// items come last.  (Reserving the places by atomics in one launch put heavy
// blocks behind light ones: triangle R-MAT-20 1.43 -> 1.7-2.5 ms.)
// Shards take the items i of entry b with (b + i + g) % shard_count ==
// shard_index; of shared items (kMerged), which begin at multiples of 8 or 16, the
// group's number counts in place of b.
struct PlanArgs {
  TrieView t;
  RevView r;
  PlanShape ps;
  uint32_t g, shard_index, shard_count;
  uint64_t* pos;    // [n_head] items (then places) of an entry: block items high, warp items low
  uint64_t* tiles;  // [tiles] sums
};
constexpr uint32_t kPlanTile = 2048;

// Neighbouring entries whose work together is small share one item (kMerged):
// its rows are looked up in their sets' lists where they lie, nothing is
// staged.  Most entries of a skewed relation end a few rows of a few candidates
// each, and an item of its own costs one of them a queue turn and a chain of
// loads of some 5,000 cycles for a hundred cycles of work (96 R-MAT graphs
// 1.77 -> 1.45 ms, lollipop Chung-Lu 2^21 4.26 -> 3.39).  Groups are aligned:
// 16 entries, or 8, of at most kMergeRows rows and kMergeElems candidates and
// elements.
constexpr uint32_t kMerged = 0x80000000u;
constexpr uint64_t kMergeRows = 128, kMergeElems = 1024;
__device__ __forceinline__ bool plan_small(const PlanArgs& p, uint32_t h0, uint32_t span) {
  if (h0 + span > p.t.n_head) return false;
  const uint64_t k0 = p.r.rev_off[h0], k1 = p.r.rev_off[h0 + span];
  return k1 - k0 <= kMergeRows && p.r.rev_wpre[k1] - p.r.rev_wpre[k0] <= kMergeElems &&
         p.t.off[h0 + span] - p.t.off[h0] <= kMergeElems;
}
// entries that share b's item, the first of which has it; 1: none
__device__ __forceinline__ uint32_t plan_span(const PlanArgs& p, uint32_t b) {
  if (!p.ps.merge) return 1;
  if (plan_small(p, b & ~15u, 16)) return 16;
  return plan_small(p, b & ~7u, 8) ? 8 : 1;
}

constexpr uint64_t kPredTrust = 4;
// items of entry b over all shards; span: plan_span
__device__ __forceinline__ uint32_t plan_items(const PlanArgs& p, uint32_t b, uint64_t k0, uint64_t k1, bool& blk,
                                               uint32_t& span) {
  blk = false;
  span = plan_span(p, b);
  if (span > 1) return (b & (span - 1)) == 0 && p.r.rev_off[b + span] > k0 ? 1 : 0;
  if (k1 <= k0) return 0;
  const uint64_t w = p.r.rev_wpre[k1] - p.r.rev_wpre[k0];
  if (p.ps.block_words && w >= kMinBlockWork) {
    const uint32_t sw = staged_words(p.t, b, p.ps.warp_words);
    blk = sw > p.ps.warp_words && sw <= p.ps.block_words;
  }
  const uint64_t mult = blk ? p.ps.warps : 1;
  const uint64_t cost = w + kRowCost * (k1 - k0);
  if (p.ps.pred) {
    // whatever the model predicts, no item of more than kPredTrust chunks: one that
    // misjudges a hub would leave it to one warp (Chung-Lu 2^20, untrained: 4.6 ms,
    // so 0.95, by chunks alone 0.70)
    const uint64_t m = (uint64_t)ceil((double)p.ps.pred[b] / (p.ps.unit * (double)mult));
    return (uint32_t)max(max((uint64_t)1, min(m, (w + 63) / 64)), cost / (kPredTrust * p.ps.chunk * mult));
  }
  return (uint32_t)((cost + p.ps.chunk * mult - 1) / (p.ps.chunk * mult));
}
// this shard's first item of entry b
__device__ __forceinline__ uint32_t plan_first(const PlanArgs& p, uint32_t b, uint32_t span) {
  return p.shard_count > 1 ? (p.shard_index + p.shard_count - (b / span + p.g) % p.shard_count) % p.shard_count : 0;
}

// zero: bytes of the control block and results to clear (a single trie, whose
// control block no copy sets up)
__global__ void __launch_bounds__(256) plan_split_kernel(PlanArgs p, Control* __restrict__ ctl, uint32_t zero) {
  __shared__ uint64_t s_warp[8];
  if (blockIdx.x == 0)
    for (uint32_t i = threadIdx.x; i < zero / 4; i += 256) reinterpret_cast<uint32_t*>(ctl)[i] = 0;
  uint64_t sum = 0;
  for (uint32_t x = threadIdx.x; x < kPlanTile; x += 256) {
    const uint64_t b = (uint64_t)blockIdx.x * kPlanTile + x;
    if (b >= p.t.n_head) break;
    bool blk;
    uint32_t span;
    const uint32_t n = plan_items(p, (uint32_t)b, p.r.rev_off[b], p.r.rev_off[b + 1], blk, span);
    const uint32_t first = plan_first(p, (uint32_t)b, span);
    const uint64_t mine = n > first ? (n - first + p.shard_count - 1) / p.shard_count : 0;
    const uint64_t v = blk ? mine << 32 : mine;
    p.pos[b] = v;
    sum += v;
  }
  sum = warp_sum(sum);
  if (lane_id() == 0) s_warp[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < 8; i++) sum += s_warp[i];
    p.tiles[blockIdx.x] = sum;
  }
}

// counts -> places in entry order; the total of this trie, and the items so far
__global__ void __launch_bounds__(256) plan_place_kernel(PlanArgs p, unsigned long long* __restrict__ total,
                                                         Control* __restrict__ ctl) {
  __shared__ uint64_t s_warp[8], s_before;
  const uint32_t lane = lane_id(), wid = threadIdx.x >> 5;
  uint64_t before = 0;  // sums of the tiles before this one
  for (uint32_t i = threadIdx.x; i < blockIdx.x; i += 256) before += p.tiles[i];
  before = warp_sum(before);
  if (lane == 0) s_warp[wid] = before;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < 8; i++) before += s_warp[i];
    s_before = before;
  }
  __syncthreads();
  before = s_before;
  const uint64_t b0 = (uint64_t)blockIdx.x * kPlanTile + 8 * threadIdx.x;
  uint64_t v[8], sum = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    v[i] = b0 + i < p.t.n_head ? p.pos[b0 + i] : 0;
    sum += v[i];
  }
  const uint64_t incl = warp_incl_scan(sum);
  if (lane == 31) s_warp[wid] = incl;
  __syncthreads();
  for (uint32_t i = 0; i < wid; i++) before += s_warp[i];
  uint64_t run = before + incl - sum;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    if (b0 + i < p.t.n_head) p.pos[b0 + i] = run;
    run += v[i];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 255) {
    *total = run;
    ctl->items[0] += (uint32_t)run;
    ctl->items[1] += (uint32_t)(run >> 32);
  }
}

// One thread per item (warp items first): item q of a class belongs to the last
// entry whose place is at or before q (entries without items share the next
// one's place and are never found), and covers the rows from the first one at
// its share of the entry's cost to the first one at the next share.  Its items
// follow those of the tries before.
__global__ void __launch_bounds__(256) plan_fill_kernel(PlanArgs p, const unsigned long long* __restrict__ total,
                                                        const Control* __restrict__ ctl, Item* __restrict__ items,
                                                        Item* __restrict__ bitems) {
  const uint32_t nw = (uint32_t)*total, nb = (uint32_t)(*total >> 32);
  const uint32_t w0 = ctl->items[0] - nw, b0 = ctl->items[1] - nb;
  for (uint64_t x = blockIdx.x * 256ull + threadIdx.x; x < (uint64_t)nw + nb; x += gridDim.x * 256ull) {
    const bool cls = x >= nw;
    const uint32_t q = cls ? (uint32_t)(x - nw) : (uint32_t)x;
    uint32_t lo = 0, hi = p.t.n_head;  // first entry with its place above q
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      const uint64_t v = __ldg(p.pos + mid);
      if ((cls ? (uint32_t)(v >> 32) : (uint32_t)v) <= q) lo = mid + 1; else hi = mid;
    }
    const uint32_t b = lo - 1;
    const uint64_t v = p.pos[b];
    const uint64_t k0 = p.r.rev_off[b], k1 = p.r.rev_off[b + 1];
    bool blk;
    uint32_t span;
    const uint64_t m = plan_items(p, b, k0, k1, blk, span);
    const uint64_t i =
        plan_first(p, b, span) + (uint64_t)(q - (cls ? (uint32_t)(v >> 32) : (uint32_t)v)) * p.shard_count;
    if (span > 1) {
      items[w0 + (nw - 1 - q)] = Item{b | kMerged, (uint32_t)k0, (uint32_t)p.r.rev_off[b + span], p.g};
      continue;
    }
    const uint64_t wp = p.r.rev_wpre[k0], W = p.r.rev_wpre[k1] - wp + kRowCost * (k1 - k0);
    const uint64_t kb = i ? row_at_cost(p.r.rev_wpre, k0, k1, wp, (W * i) / m) : k0;
    const uint64_t ke = i + 1 < m ? row_at_cost(p.r.rev_wpre, k0, k1, wp, (W * (i + 1)) / m) : k1;
    (cls ? bitems + b0 + (nb - 1 - q) : items + w0 + (nw - 1 - q))[0] = Item{b, (uint32_t)kb, (uint32_t)ke, p.g};
  }
}

// L2 eviction priority for the word rows' loads of N(a)'s bitset words: the
// sources of the word rows are the density rule's dense sets (75 MB of words
// at R-MAT-22, each read ~130 times in a query), so they are kept ahead of the
// streamed candidate values (createpolicy + ld.global.nc.L2::cache_hint).
__device__ __forceinline__ uint64_t l2_policy_last() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ ulonglong2 ld2_hint(const uint64_t* a, uint64_t pol) {
  ulonglong2 v;
  asm("ld.global.nc.L2::cache_hint.v2.u64 {%0, %1}, [%2], %3;" : "=l"(v.x), "=l"(v.y) : "l"(a), "l"(pol));
  return v;
}
__device__ __forceinline__ uint64_t ld64_hint(const uint64_t* a, uint64_t pol) {
  uint64_t v;
  asm("ld.global.nc.L2::cache_hint.u64 %0, [%1], %2;" : "=l"(v) : "l"(a), "l"(pol));
  return v;
}
// ------------------------------------------------------------------ probes
// Probe structures for the staged set N(b), one per stored layout.
// P_ZBITS: a range bitset too large to stage word for word, staged
// compressed: per group of 32 words a presence mask (bit i: word 32k + i is
// non-zero) beside the count of non-zero words before the group, read
// together in one 8-byte load, and then only the non-zero words.  A probe
// whose word is empty costs one shared load; the others two.
enum { P_SBITS = 0, P_GBITS = 1, P_SLIST = 2, P_GLIST = 3, P_GBLOCK = 4, P_ZBITS = 5 };

struct Staged {
  const uint64_t* words;  // P_SBITS (shared) / P_GBITS (global); P_ZBITS: the non-zero words (shared)
  const uint32_t* list;   // P_SLIST (shared) / P_GLIST (global)
  const uint32_t* ids;    // P_GBLOCK
  const uint64_t* bwords; // P_GBLOCK
  const uint2* pz;        // P_ZBITS: group k: x = presence mask of words 32k.., y = non-zero words before 32k
  uint32_t start;         // first word index (bitsets)
  uint32_t n;             // words / list length / blocks
};


// branch-free lower bound over a sorted run of n >= 1 values
template <bool kShared>
__device__ __forceinline__ bool list_contains(const uint32_t* p, uint32_t n, uint32_t w) {
  uint32_t base = 0;
  while (n > 1) {
    const uint32_t half = n >> 1;
    const uint32_t v = kShared ? p[base + half] : __ldg(p + base + half);
    base = (v <= w) ? base + half : base;
    n -= half;
  }
  return (kShared ? p[base] : __ldg(p + base)) == w;
}

template <int P>
__device__ __forceinline__ uint32_t probe(const Staged& s, uint32_t w) {
  if (P == P_ZBITS) {
    const uint32_t idx = (w >> 6) - s.start;
    if (idx >= s.n) return 0;  // also catches w below the first word (wraps)
    const uint2 g = s.pz[idx >> 5];
    if (!((g.x >> (idx & 31)) & 1u)) return 0;
    const uint32_t below = g.x & ((1u << (idx & 31)) - 1u);
    return (uint32_t)(s.words[g.y + __popc(below)] >> (w & 63)) & 1u;
  }
  if (P == P_SBITS || P == P_GBITS) {
    const uint32_t idx = (w >> 6) - s.start;
    if (idx >= s.n) return 0;  // also catches w below the first word (wraps)
    const uint64_t word = (P == P_SBITS) ? s.words[idx] : __ldg(s.words + idx);
    return (uint32_t)(word >> (w & 63)) & 1u;
  } else if (P == P_SLIST || P == P_GLIST) {
    return list_contains<P == P_SLIST>(s.list, s.n, w) ? 1u : 0u;
  } else {  // block bitset: find block id w >> 8, test its word
    const uint32_t id = w >> 8;
    uint32_t lo = 0, hi = s.n;
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (__ldg(s.ids + mid) < id) lo = mid + 1; else hi = mid;
    }
    if (lo >= s.n || __ldg(s.ids + lo) != id) return 0;
    return (uint32_t)(__ldg(s.bwords + 4 * (uint64_t)lo + ((w >> 6) & 3)) >> (w & 63)) & 1u;
  }
}

// What a hit does besides counting: kMode 0 counts only; 1 adds it to the
// annotation of the row's source (and, on a symmetric relation, of the
// matched element) -- the annotated bag of TrieBuilder::set_annotation;
// 2 writes the tuple (a, b, c) to the item's slice of the output columns
// -- the materialized Triangle(a,b,c) of TrieBuilder::build_set.
enum { MODE_COUNT = 0, MODE_ANNOT = 1, MODE_MAT = 2 };

constexpr int kHot = 4;  // MODE_ANNOT: head entries with block-local counters
struct Int4 {
  int32_t v[kHot];
};

struct Sink {
  unsigned long long* annot;  // MODE_ANNOT
  uint32_t* ma;               // MODE_MAT: output columns
  uint32_t* mb;
  uint32_t* mc;
  uint64_t base;              // MODE_MAT: first row of this item's slice
  unsigned int* slot;         // MODE_MAT: the warp's running row count (shared)
  uint32_t b;                 // MODE_MAT: value of the staged head entry b
  const int32_t* hot;         // MODE_ANNOT: the kHot largest sets' head entries (-1: none)
  unsigned long long* hot_acc;  // MODE_ANNOT: their block-local counts (shared)
  // MODE_ANNOT on a symmetric relation: every matched element is in the
  // staged N(b); when it is staged with room to spare, each element has a
  // shared counter (wcnt, by position in N(b)) flushed once per item
  uint32_t* wcnt;             // null: matched elements go to the annotation directly
  int wmode;                  // P_SLIST (position by search) or P_SBITS (position by rank)
  const uint32_t* wlist;      // P_SLIST: the staged list, wn elements
  const uint64_t* wwords;     // P_SBITS: the staged words, wn of them from word wstart
  const uint32_t* wrank;      // P_SBITS: staged elements before each staged word
  uint32_t wstart, wn;
};

// owner lane of flattened pair q: the number of lanes whose inclusive
// prefix is <= q (q < total guarantees a result below 32)
__device__ __forceinline__ uint32_t owner_lane(uint32_t incl, uint32_t q) {
  uint32_t j = 0;
#pragma unroll
  for (int step = 16; step; step >>= 1) {
    const uint32_t tj = __shfl_sync(kFull, incl, j + step - 1);
    if (tj <= q) j += step;
  }
  return j;
}

// kSrcAgg: the caller adds the row source's share of the annotation for a
// run of hits at once (add_src), so a hit adds only the matched element's
// share; a hub source in many rows would otherwise take one atomic per hit.
template <int kMode, bool kSrcAgg = false>
__device__ __forceinline__ void on_hit(const TrieView& t, const RevView& r, const Sink& sk, uint32_t src,
                                       uint32_t w) {
  if (kMode == MODE_ANNOT) {
    if (r.dir == DIR_SYM) {
      if (!kSrcAgg) atomicAdd(sk.annot + src, 2ull);
      if (sk.wcnt) {  // the matched element's position in the staged N(b)
        uint32_t pos;
        if (sk.wmode == P_SLIST) {
          uint32_t lo = 0, hi = sk.wn;
          while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (sk.wlist[mid] < w) lo = mid + 1; else hi = mid;
          }
          pos = lo;
        } else {
          const uint32_t idx = (w >> 6) - sk.wstart;
          pos = sk.wrank[idx] + (uint32_t)__popcll(sk.wwords[idx] & ((1ull << (w & 63)) - 1));
        }
        atomicAdd(sk.wcnt + pos, 1u);
        return;
      }
      // the matched element: a hub is the third vertex of a large share of
      // all triangles, so the largest sets count in shared memory first
      const int32_t hx = __ldg(t.head_index + w);
      int k = 0;
#pragma unroll
      for (; k < kHot; k++)
        if (hx == sk.hot[k]) break;
      if (k < kHot) atomicAdd(sk.hot_acc + k, 2ull);
      else atomicAdd(sk.annot + hx, 2ull);
    } else if (!kSrcAgg) {
      atomicAdd(sk.annot + src, 1ull);
    }
  } else if (kMode == MODE_MAT) {
    const uint32_t a = __ldg(t.head + src), b = sk.b;
    if (r.dir == DIR_SYM) {
      // one undirected triangle a < b < w stands for all 3! orderings
      const uint64_t o = sk.base + atomicAdd(sk.slot, 6u);
      const uint32_t p[6][3] = {{a, b, w}, {a, w, b}, {b, a, w}, {b, w, a}, {w, a, b}, {w, b, a}};
#pragma unroll
      for (int k = 0; k < 6; k++) {
        sk.ma[o + k] = p[k][0];
        sk.mb[o + k] = p[k][1];
        sk.mc[o + k] = p[k][2];
      }
    } else {
      const uint64_t o = sk.base + atomicAdd(sk.slot, 1u);
      sk.ma[o] = a;
      sk.mb[o] = b;
      sk.mc[o] = w;
    }
  }
}

template <int kMode>
__device__ __forceinline__ void add_src(const RevView& r, const Sink& sk, uint32_t src, uint64_t hits) {
  if (kMode == MODE_ANNOT && hits) atomicAdd(sk.annot + src, (r.dir == DIR_SYM ? 2ull : 1ull) * hits);
}

// Rows whose source set N(a) is also a range bitset, against a bitset N(b),
// are intersected word by word (64-bit AND + popcount over the overlap of
// the candidate value range [v0, v1] with both word ranges) whenever the
// words, weighted by kWordRowNum / kWordRowDen (a word against a candidate
// probe), are fewer than the row's candidate elements; the reference's
// bitset ∩ bitset path (ops/intersection/bitset.hpp:526-567, 619-661).
// Word rows run warp-cooperatively one row at a time (coalesced 8-byte
// loads of N(a)'s words); the other rows are flattened (row, element)
// pairs over the lanes, two pairs per lane per trip for memory-level
// parallelism.
template <int P, int kMode>
__device__ __forceinline__ uint64_t stream_rows(const Staged& st, const TrieView& t, const RevView& r, uint32_t kb,
                                                uint32_t ke, uint32_t long_row, const Sink& sk) {
  constexpr bool kBits = (P == P_SBITS || P == P_GBITS);
  const uint32_t lane = lane_id();
  uint64_t cnt = 0;
  const uint64_t pol_keep = l2_policy_last();
  for (uint32_t k0 = kb; k0 < ke; k0 += 32) {
    const uint32_t k = k0 + lane;
    uint32_t lo = 0, len = 0, src = 0;
    if (k < ke) {
      lo = __ldg(r.rev_lo + k);
      len = __ldg(r.rev_hi + k) - lo;
      src = __ldg(r.rev_src + k);
    }
    // ---- word rows
    if (kBits) {
      bool word_row = false;
      uint32_t v0 = 0, v1 = 0, wlo = 0, whi = 0;
      uint64_t abase = 0;
      if (len && __ldg(t.layout + src) == EH_LAYOUT_RANGE_BITSET) {
        v0 = __ldg(t.vals + lo);
        v1 = __ldg(t.vals + lo + len - 1);
        const SetAux aa = t.aux[src];
        const uint32_t lo_w = max(max(v0 >> 6, aa.start), st.start);
        const uint32_t hi_w = min(min(v1 >> 6, aa.start + aa.n - 1), st.start + st.n - 1);
        const uint32_t words = hi_w >= lo_w ? hi_w - lo_w + 1 : 0;
        if (words * kWordRowNum < len * kWordRowDen) {
          word_row = true;
          wlo = lo_w;
          whi = hi_w;
          abase = aa.off - aa.start;  // word w of N(a) is bs_words[abase + w]
        }
      }
      uint32_t nw = (word_row && whi >= wlo) ? whi - wlo + 1 : 0u;
      if (word_row) len = 0;  // handled here, not in the element loop
      // long word rows (at least a warp's width of words): one row at a time
      // across the warp, each lane ANDing the word pairs 2 lane, 2 lane + 64,
      // ... read from N(a) with one aligned 16-byte load (the reference's
      // 128-bit AND), no owner search
      {
        const bool is_long = nw >= (uint32_t)kLongWords;
        uint32_t rows = __ballot_sync(kFull, is_long);
        if (is_long) nw = 0;
        while (rows) {
          const int j = __ffs(rows) - 1;
          rows &= rows - 1;
          const uint32_t lo_w = __shfl_sync(kFull, wlo, j), hi_w = __shfl_sync(kFull, whi, j);
          const uint32_t b0 = __shfl_sync(kFull, v0, j), b1 = __shfl_sync(kFull, v1, j);
          const uint64_t base = __shfl_sync(kFull, abase, j);
          const uint32_t sj = __shfl_sync(kFull, src, j);
          const uint32_t w_first = b0 >> 6, w_last = b1 >> 6;
          uint32_t row_hits = 0;
          // The row's words lo_w..hi_w are read in pairs from an even pool
          // index, 16-byte aligned (allocations are at least 16-byte
          // aligned): pair q holds the row's words q - par and q + 1 - par,
          // where par = 1 when the row starts at an odd pool index (its first
          // pair then begins with the word before lo_w: in the pool, since
          // that index is >= 1, and masked).  Offsets stay non-negative; a
          // word index is formed only for words inside the row.  A pair is
          // read whole only when both its words are in the row's range or the
          // first one is the word before it, so no read passes N(a)'s last word.
          const uint32_t par = (uint32_t)((base + lo_w) & 1ull);
          const uint32_t end = hi_w - lo_w + 1 + par;         // pair offsets run below end
          const uint64_t g0 = base + lo_w - par;              // even pool index of offset 0
          const uint32_t wa = lo_w - par;                     // word of offset 0 (mod 2^32)
          const uint32_t sa = wa - st.start;                  // its staged index (mod 2^32)
          for (uint32_t q0 = 2 * lane; q0 < end; q0 += 64 * kLongWordUnroll) {
            uint64_t x[2 * kLongWordUnroll], y[2 * kLongWordUnroll];
#pragma unroll
            for (int u = 0; u < kLongWordUnroll; u++) {
              const uint32_t q = q0 + 64 * u;
              if (q + 2 <= end) {
                const ulonglong2 v = ld2_hint(t.bs_words + g0 + q, pol_keep);
                x[2 * u] = v.x;
                x[2 * u + 1] = v.y;
              } else {
                x[2 * u] = q < end ? ld64_hint(t.bs_words + g0 + q, pol_keep) : 0ull;
                x[2 * u + 1] = 0ull;
              }
#pragma unroll
              for (int h = 0; h < 2; h++) {
                const uint32_t qh = q + h;
                const bool in = qh >= par && qh < end;  // a word of the row
                y[2 * u + h] = in ? ((P == P_SBITS) ? st.words[sa + qh] : __ldg(st.words + (sa + qh))) : 0ull;
              }
            }
#pragma unroll
            for (int u = 0; u < 2 * kLongWordUnroll; u++) {
              const uint32_t w = wa + (q0 + 64 * (u >> 1) + (u & 1));  // meaningful where y is non-zero
              if (w == w_first) y[u] &= ~0ull << (b0 & 63);
              if (w == w_last) y[u] &= ~0ull >> (63 - (b1 & 63));
              x[u] &= y[u];
              row_hits += __popcll(x[u]);
            }
            if (kMode == MODE_MAT || (kMode == MODE_ANNOT && r.dir == DIR_SYM)) {
#pragma unroll
              for (int u = 0; u < 2 * kLongWordUnroll; u++) {
                uint64_t z = x[u];  // non-zero only for words inside the row
                const uint32_t w = wa + (q0 + 64 * (u >> 1) + (u & 1));
                while (z) {
                  const uint32_t bit = __ffsll((long long)z) - 1;
                  on_hit<kMode, true>(t, r, sk, sj, (w << 6) | bit);
                  z &= z - 1;
                }
              }
            }
          }
          cnt += row_hits;
          if (kMode == MODE_ANNOT) {  // the row's source once per row
            const uint32_t rh = warp_sum(row_hits);
            if (lane == 0) add_src<kMode>(r, sk, sj, rh);
          }
        }
      }
      // the other word rows of this batch, flattened into (row, word) pairs
      // over the lanes like the short element rows below: one trip covers
      // the words of many rows
      const uint32_t wincl = warp_incl_scan(nw);
      const uint32_t wtotal = __shfl_sync(kFull, wincl, 31);
      const uint32_t wexcl = wincl - nw;
      for (uint32_t p = 0; p < wtotal; p += 32 * kWordUnroll) {
        uint64_t x[kWordUnroll];
        uint32_t wv[kWordUnroll], sj[kWordUnroll];
#pragma unroll
        for (int u = 0; u < kWordUnroll; u++) {
          const uint32_t q = p + 32 * u + lane;
          const uint32_t j = owner_lane(wincl, q);
          const uint32_t lo_w = __shfl_sync(kFull, wlo, j), ex = __shfl_sync(kFull, wexcl, j);
          const uint32_t b0 = __shfl_sync(kFull, v0, j), b1 = __shfl_sync(kFull, v1, j);
          const uint64_t base = __shfl_sync(kFull, abase, j);
          sj[u] = __shfl_sync(kFull, src, j);
          x[u] = 0;
          wv[u] = 0;
          if (q < wtotal) {
            const uint32_t w = lo_w + (q - ex);
            uint64_t m = ~0ull;
            if (w == (b0 >> 6)) m &= ~0ull << (b0 & 63);
            if (w == (b1 >> 6)) m &= ~0ull >> (63 - (b1 & 63));
            const uint64_t bw = (P == P_SBITS) ? st.words[w - st.start] : __ldg(st.words + (w - st.start));
            x[u] = ld64_hint(t.bs_words + base + w, pol_keep) & bw & m;
            wv[u] = w;
          }
        }
#pragma unroll
        for (int u = 0; u < kWordUnroll; u++) {
          const uint32_t hits = __popcll(x[u]);
          cnt += hits;
          if (kMode == MODE_ANNOT) add_src<kMode>(r, sk, sj[u], hits);
          if (kMode == MODE_MAT || (kMode == MODE_ANNOT && r.dir == DIR_SYM)) {
            uint64_t y = x[u];
            while (y) {
              const uint32_t bit = __ffsll((long long)y) - 1;
              on_hit<kMode, true>(t, r, sk, sj[u], (wv[u] << 6) | bit);
              y &= y - 1;
            }
          }
        }
      }
    }
    // ---- long element rows: two rows at a time across the warp, each lane
    // loading kLongUnroll coalesced elements of both before it probes any,
    // no owner search
    {
      const bool is_long = len >= long_row;
      uint32_t rows = __ballot_sync(kFull, is_long);
      const uint32_t rlen = len;
      if (is_long) len = 0;
      while (rows) {
        const int j = __ffs(rows) - 1;
        rows &= rows - 1;
        int j2 = j;
        bool two = false;
        if (rows) {
          j2 = __ffs(rows) - 1;
          rows &= rows - 1;
          two = true;
        }
        const uint32_t rlo = __shfl_sync(kFull, lo, j), rn = __shfl_sync(kFull, rlen, j);
        const uint32_t rlo2 = __shfl_sync(kFull, lo, j2);
        const uint32_t rn2 = two ? __shfl_sync(kFull, rlen, j2) : 0u;
        const uint32_t src_j = __shfl_sync(kFull, src, j), src_j2 = __shfl_sync(kFull, src, j2);
        const uint32_t* row = t.vals + rlo;
        const uint32_t* row2 = t.vals + rlo2;
        uint32_t row_hits = 0, row_hits2 = 0;
        const uint32_t rmax = rn > rn2 ? rn : rn2;
        for (uint32_t i = lane; i < rmax; i += 32 * kLongUnroll) {
          uint32_t w[kLongUnroll], w2[kLongUnroll];
#pragma unroll
          for (int u = 0; u < kLongUnroll; u++) {
            w[u] = (i + 32 * u < rn) ? __ldg(row + i + 32 * u) : 0u;
            w2[u] = (i + 32 * u < rn2) ? __ldg(row2 + i + 32 * u) : 0u;
          }
#pragma unroll
          for (int u = 0; u < kLongUnroll; u++) {
            if (i + 32 * u < rn) {
              const uint32_t h = probe<P>(st, w[u]);
              row_hits += h;
              if (h) on_hit<kMode, true>(t, r, sk, src_j, w[u]);
            }
            if (i + 32 * u < rn2) {
              const uint32_t h = probe<P>(st, w2[u]);
              row_hits2 += h;
              if (h) on_hit<kMode, true>(t, r, sk, src_j2, w2[u]);
            }
          }
        }
        cnt += row_hits + row_hits2;
        if (kMode == MODE_ANNOT) {  // each row's source once per row
          const uint32_t rh = warp_sum(row_hits);
          const uint32_t rh2 = warp_sum(row_hits2);
          if (lane == 0) {
            add_src<kMode>(r, sk, src_j, rh);
            if (two) add_src<kMode>(r, sk, src_j2, rh2);
          }
        }
      }
    }
    // ---- short element rows, flattened
    const uint32_t incl = warp_incl_scan(len);
    const uint32_t total = __shfl_sync(kFull, incl, 31);
    const uint32_t excl = incl - len;
    for (uint32_t p = 0; p < total; p += 32 * kShortUnroll) {
      uint32_t w[kShortUnroll], sj[kShortUnroll];
#pragma unroll
      for (int u = 0; u < kShortUnroll; u++) {
        const uint32_t q = p + 32 * u + lane;
        const uint32_t j = owner_lane(incl, q);
        const uint32_t loj = __shfl_sync(kFull, lo, j), exj = __shfl_sync(kFull, excl, j);
        sj[u] = __shfl_sync(kFull, src, j);
        w[u] = q < total ? __ldg(t.vals + loj + (q - exj)) : 0u;
      }
#pragma unroll
      for (int u = 0; u < kShortUnroll; u++) {
        const uint32_t q = p + 32 * u + lane;
        const uint32_t h = q < total ? probe<P>(st, w[u]) : 0u;
        cnt += h;
        if (kMode == MODE_ANNOT) {
          // lanes of one row are adjacent: one source atomic per row present
          const uint32_t grp = __match_any_sync(kFull, sj[u]);
          const uint32_t hm = __ballot_sync(kFull, h) & grp;
          if (lane == (uint32_t)(__ffs(grp) - 1)) add_src<kMode>(r, sk, sj[u], __popc(hm));
        }
        if (h) on_hit<kMode, true>(t, r, sk, sj[u], w[u]);
      }
    }
  }
  return cnt;
}

// probe() for bit words, on their 32-bit halves: these passes are bound by
// instruction issue, and a 64-bit variable shift takes several
template <int P>
__device__ __forceinline__ bool hit(const Staged& st, uint32_t w) {
  if (P == P_SBITS || P == P_GBITS) {
    const uint32_t idx = (w >> 5) - 2 * st.start;
    if (idx >= 2 * st.n) return false;  // also below the first word (wraps)
    const uint32_t* h = reinterpret_cast<const uint32_t*>(st.words) + idx;
    return ((P == P_SBITS ? *h : __ldg(h)) >> (w & 31)) & 1u;
  }
  if (P == P_ZBITS) {
    const uint32_t idx = (w >> 6) - st.start;
    if (idx >= st.n) return false;
    const uint2 g = st.pz[idx >> 5];
    const uint32_t up = g.x >> (idx & 31);
    if (!(up & 1u)) return false;
    const uint32_t pos = g.y + __popc(g.x ^ (up << (idx & 31)));
    return (reinterpret_cast<const uint32_t*>(st.words)[2 * pos + ((w >> 5) & 1u)] >> (w & 31)) & 1u;
  }
  return probe<P>(st, w) != 0;
}

// stream_rows for the plain COUNT.  A batch of 32 rows, a row per lane; each
// row is counted in one of five ways:
//   word trips     both sets are range bitsets and their common words are fewer
//                  than the candidates (weighted as in stream_rows), at least
//                  kTripWords of them: 32 words per trip
//   word pairs     fewer words: flattened (row, word) pairs over the lanes
//   wide rows      at least kWideRow candidates: the warp runs along the row, no trip
//                  to be looked up
//   element trips  at least long_row candidates: 32 candidates per trip
//   element pairs  fewer: flattened (row, candidate) pairs over the lanes
// The trips of all rows of a batch form one list, taken kTrips at a time with
// their loads issued before the first is used, so that a row need not fill
// them; the trip's row is found by one ballot.  A word row needs no masks: what
// N(a) holds outside the candidates is at or before b (after, on a relation
// that goes down), where N(b) holds nothing -- or, on a symmetric relation, the
// staged copy of N(b) had it cleared -- so neither its first nor its last
// candidate is read.
// Measured (triangle kernel, R-MAT-22 / R-MAT-20, ms): stream_rows 8.49 / 1.43;
// trips of four 8.10 / 1.21; views as kernel parameters and the next batch's
// rows loaded ahead 7.76 / 1.14; element trips by eight 7.18 / 1.13 (by six
// 7.29, word trips by three 7.40, by six 7.39).  48 registers and five blocks per
// SM 7.84, 80 and three 9.41.  Wide rows apart from 128 / 256 / 512 / 1024 candidates
// or never: R-MAT-22 6.95 / 6.59 / 6.67 / 6.67 / 6.67, Chung-Lu 2^18 by descending
// degree 5.35 / 5.36 / 5.43 / 5.57 / 7.85, Chung-Lu 2^21 1.66 / 1.65 / 1.70 / 1.70 /
// 1.70 (a trip costs a ballot and two shuffles per 32 candidates: a star's rows ran
// at 2.35 instead of 1.23).
constexpr int kTrips = 8, kWTrips = 4;
constexpr uint32_t kTripWords = 16, kWideRow = 256;
template <int P>
__device__ __forceinline__ uint64_t count_rows(const Staged& st, const TrieView& t, const RevView& r, uint32_t kb,
                                               uint32_t ke, uint32_t long_row) {
  const uint32_t lane = lane_id();
  // unstaged words of a symmetric N(b) are not cleared: element rows only
  const bool words_ok = P == P_SBITS || (P == P_GBITS && !t.up);
  const uint64_t pol_keep = l2_policy_last();
  constexpr bool kWords = P == P_SBITS || P == P_GBITS;
  uint64_t total_hits = 0;
  uint32_t next_lo = 0, next_hi = 0, next_src = 0;  // the next batch's rows, loaded a batch ahead
  if (kb + lane < ke) {
    next_lo = __ldg(r.rev_lo + kb + lane);
    next_hi = __ldg(r.rev_hi + kb + lane);
    if (kWords) next_src = __ldg(r.rev_src + kb + lane);
  }
  for (uint32_t k0 = kb; k0 < ke; k0 += 32) {
    const uint32_t lo = next_lo, src = next_src;
    uint32_t len = next_hi - next_lo;
    next_lo = next_hi = 0;
    if (k0 + 32 + lane < ke) {
      next_lo = __ldg(r.rev_lo + k0 + 32 + lane);
      next_hi = __ldg(r.rev_hi + k0 + 32 + lane);
      if (kWords) next_src = __ldg(r.rev_src + k0 + 32 + lane);
    }
    uint32_t cnt = 0;
    uint32_t nw = 0, ws = 0;   // words of a word row; its first one, from N(b)'s start
    uint64_t wbase = 0;        // and in the pool
    if (kWords && words_ok && len && __ldg(t.layout + src) == EH_LAYOUT_RANGE_BITSET) {
      const SetAux aa = t.aux[src];
      const uint32_t lo_w = max(aa.start, st.start);
      const uint32_t hi_w = min(aa.start + aa.n, st.start + st.n);
      const uint32_t words = hi_w > lo_w ? hi_w - lo_w : 0;
      if (words * kWordRowNum < len * kWordRowDen) {
        len = 0;
        nw = words;
        ws = lo_w - st.start;
        wbase = aa.off + (lo_w - aa.start);
      }
    }
    if (kWords) {
      const uint32_t nt = nw >= kTripWords ? (nw + 31) >> 5 : 0;
      const uint32_t incl = warp_incl_scan(nt);
      const uint32_t total = __shfl_sync(kFull, incl, 31);
      if (total) {
        const uint32_t first = 32 * (incl - nt);  // word q of the list is word q - first of its row
        const uint64_t pool = wbase - first;
        const uint32_t staged = ws - first, end = nw + first;
        for (uint32_t t0 = 0; t0 < total; t0 += kWTrips) {
          uint64_t x[kWTrips], y[kWTrips];
#pragma unroll
          for (int u = 0; u < kWTrips; u++) {
            const uint32_t trip = min(t0 + u, total - 1);
            const int j = __popc(__ballot_sync(kFull, incl <= trip));
            const uint32_t q = 32 * trip + lane;
            const uint64_t pj = __shfl_sync(kFull, pool, j);
            const uint32_t sj = __shfl_sync(kFull, staged, j), ej = __shfl_sync(kFull, end, j);
            const bool in = q < ej && t0 + u < total;
            x[u] = in ? ld64_hint(t.bs_words + (pj + q), pol_keep) : 0ull;
            y[u] = in ? ((P == P_SBITS) ? st.words[sj + q] : __ldg(st.words + (sj + q))) : 0ull;
          }
#pragma unroll
          for (int u = 0; u < kWTrips; u++) cnt += __popcll(x[u] & y[u]);
        }
        if (nt) nw = 0;
      }
      const uint32_t wincl = warp_incl_scan(nw);
      const uint32_t wtotal = __shfl_sync(kFull, wincl, 31);
      const uint32_t wfirst = wincl - nw;
      const uint64_t wpool = wbase - wfirst;
      const uint32_t wstaged = ws - wfirst;
      for (uint32_t p = 0; p < wtotal; p += 64) {
        uint64_t x[2], y[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
          const uint32_t q = p + 32 * u + lane;
          const uint32_t j = owner_lane(wincl, min(q, wtotal - 1));
          const uint64_t pj = __shfl_sync(kFull, wpool, j);
          const uint32_t sj = __shfl_sync(kFull, wstaged, j);
          x[u] = q < wtotal ? ld64_hint(t.bs_words + (pj + q), pol_keep) : 0ull;
          y[u] = q < wtotal ? ((P == P_SBITS) ? st.words[sj + q] : __ldg(st.words + (sj + q))) : 0ull;
        }
        cnt += __popcll(x[0] & y[0]) + __popcll(x[1] & y[1]);
      }
    }
    for (uint32_t rows = __ballot_sync(kFull, len >= kWideRow); rows; rows &= rows - 1) {
      const int j = __ffs(rows) - 1;
      const uint32_t* row = t.vals + __shfl_sync(kFull, lo, j);
      const uint32_t n = __shfl_sync(kFull, len, j);
      uint32_t i = lane;
      for (; i + 32 * (kTrips - 1) < n; i += 32 * kTrips) {
        uint32_t v[kTrips];
#pragma unroll
        for (int u = 0; u < kTrips; u++) v[u] = __ldg(row + (i + 32 * u));
#pragma unroll
        for (int u = 0; u < kTrips; u++) cnt += hit<P>(st, v[u]);
      }
      for (; i < n; i += 32) cnt += hit<P>(st, __ldg(row + i));
      if (lane == j) len = 0;
    }
    {
      const uint32_t nt = len >= long_row ? (len + 31) >> 5 : 0;
      const uint32_t incl = warp_incl_scan(nt);
      const uint32_t total = __shfl_sync(kFull, incl, 31);
      if (total) {
        const uint32_t first = 32 * (incl - nt);
        const uint32_t elem = lo - first, end = len + first;
        for (uint32_t t0 = 0; t0 < total; t0 += kTrips) {
          uint32_t v[kTrips];
          bool in[kTrips];
#pragma unroll
          for (int u = 0; u < kTrips; u++) {
            const uint32_t trip = min(t0 + u, total - 1);
            const int j = __popc(__ballot_sync(kFull, incl <= trip));
            const uint32_t q = 32 * trip + lane;
            const uint32_t ej = __shfl_sync(kFull, elem, j);
            in[u] = q < __shfl_sync(kFull, end, j) && t0 + u < total;
            v[u] = in[u] ? __ldg(t.vals + (ej + q)) : 0u;
          }
#pragma unroll
          for (int u = 0; u < kTrips; u++) cnt += in[u] && hit<P>(st, v[u]);
        }
        if (nt) len = 0;
      }
    }
    const uint32_t incl = warp_incl_scan(len);
    const uint32_t total = __shfl_sync(kFull, incl, 31);
    const uint32_t elem = lo - (incl - len);
    for (uint32_t p = 0; p < total; p += 32 * kShortUnroll) {
      uint32_t v[kShortUnroll];
#pragma unroll
      for (int u = 0; u < kShortUnroll; u++) {
        const uint32_t q = p + 32 * u + lane;
        const uint32_t j = owner_lane(incl, min(q, total - 1));
        const uint32_t ej = __shfl_sync(kFull, elem, j);
        v[u] = q < total ? __ldg(t.vals + (ej + q)) : 0u;
      }
#pragma unroll
      for (int u = 0; u < kShortUnroll; u++) cnt += p + 32 * u + lane < total && hit<P>(st, v[u]);
    }
    total_hits += cnt;  // a batch's hits per lane stay far below 2^32
  }
  return total_hits;
}

// Entries of a merged item: lane i <= 15 holds entry h0 + i's first row and its
// staged range (entries past the item's last row are never asked for).
struct Merged {
  uint64_t s0;
  uint32_t len, row;
  __device__ __forceinline__ Merged(const TrieView& t, const RevView& r, uint32_t h0) {
    const uint32_t i = lane_id() & 15u;
    const uint32_t h = min(h0 + i, t.n_head - 1);
    const StagedRange sr = staged_range(t, h);
    s0 = sr.s0;
    len = sr.len;
    row = h0 + i < t.n_head ? (uint32_t)__ldg(r.rev_off + h) : 0xffffffffu;
  }
  // which entry row k belongs to: the last one that starts at or before it
  __device__ __forceinline__ uint32_t entry(uint32_t k) const {
    uint32_t e = 0;
#pragma unroll
    for (int step = 8; step; step >>= 1) {
      const uint32_t v = __shfl_sync(kFull, row, e + step);
      if (v <= k) e += step;
    }
    return e;
  }
};
__device__ __forceinline__ bool list_has(const uint32_t* __restrict__ vals, uint32_t s0, uint32_t n, uint32_t w) {
  const uint32_t* p = vals + s0;  // n >= 1: an entry with rows has a staged part
  while (n > 1) {
    const uint32_t half = n >> 1;
    if (__ldg(p + half) <= w) p += half;
    n -= half;
  }
  return __ldg(p) == w;
}
// the hits of a merged item: flattened (row, candidate) pairs, each looked up in
// its own entry's list
__device__ __forceinline__ uint32_t count_merged(const TrieView& t, const RevView& r, uint32_t h0, uint32_t kb,
                                                 uint32_t ke) {
  const uint32_t lane = lane_id();
  const Merged m(t, r, h0);
  uint32_t cnt = 0;
  for (uint32_t k0 = kb; k0 < ke; k0 += 32) {
    const uint32_t k = k0 + lane;
    uint32_t lo = 0, len = 0;
    if (k < ke) {
      lo = __ldg(r.rev_lo + k);
      len = __ldg(r.rev_hi + k) - lo;
    }
    const uint32_t e = m.entry(min(k, ke - 1));
    const uint32_t s0 = __shfl_sync(kFull, (uint32_t)m.s0, e), n = __shfl_sync(kFull, m.len, e);
    const uint32_t incl = warp_incl_scan(len);
    const uint32_t total = __shfl_sync(kFull, incl, 31);
    const uint32_t elem = lo - (incl - len);
    for (uint32_t p = 0; p < total; p += 64) {
      uint32_t w[2], sj[2], nj[2];
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const uint32_t q = min(p + 32 * u + lane, total - 1);
        const uint32_t j = owner_lane(incl, q);
        w[u] = __ldg(t.vals + (__shfl_sync(kFull, elem, j) + q));
        sj[u] = __shfl_sync(kFull, s0, j);
        nj[u] = __shfl_sync(kFull, n, j);
      }
#pragma unroll
      for (int u = 0; u < 2; u++) cnt += p + 32 * u + lane < total && list_has(t.vals, sj[u], nj[u], w[u]);
    }
  }
  return cnt;
}

__device__ __forceinline__ bool few_candidates(const RevView& r, const Item& item) {
  return item.ke - item.kb <= kListRows &&
         __ldg(r.rev_wpre + item.ke) - __ldg(r.rev_wpre + item.kb) <= kListCandidates;
}

// The annotated pass's rows run longer on a list than count_rows', so a bitmap has to
// serve more of them (kernel ms, from 1,000 / 3,000 / 10,000 candidates, lists always:
// R-MAT-20 of edge factor 4 by its own ids, down 2.94 / 3.00 / 2.62, 2.65, general 9.4 /
// 9.3 / 9.0, 8.5; Chung-Lu 2^20 of exponent 2.6, general 8.0 / 8.0 / 7.3, 7.4; R-MAT-16,
// general 1.37 / 1.42 / 1.88, 1.95).
constexpr uint64_t kAnnotCandidates = 10000;
__device__ __forceinline__ bool many_candidates(const RevView& r, const Item& item) {
  return __ldg(r.rev_wpre + item.ke) - __ldg(r.rev_wpre + item.kb) >= kAnnotCandidates;
}

// Stage N(b) in the warp's shared region according to its layout; returns
// the probe mode.  zlist: lists as bitmaps; blocks_too: block bitsets that fit as lists
// as well, by their elements.
__device__ __forceinline__ int stage_set(const TrieView& t, uint32_t hb, uint32_t* sm, int cap_words, Staged& st,
                                         bool zlist = false, bool blocks_too = false) {
  const uint32_t lane = lane_id();
  const uint8_t layout = t.layout[hb];
  const StagedRange sr = staged_range(t, hb);
  const uint64_t s0 = sr.s0;
  const uint32_t len = sr.len;
  const SetAux a = layout == EH_LAYOUT_RANGE_BITSET ? staged_bits(t, hb, sr) : t.aux[hb];
  if (layout == EH_LAYOUT_RANGE_BITSET) {
    st.start = a.start;
    st.n = a.n;
    if (2 * a.n <= (uint32_t)cap_words) {
      uint64_t* sw = reinterpret_cast<uint64_t*>(sm);
      for (uint32_t j = lane; j < a.n; j += 32) sw[j] = __ldg(t.bs_words + a.off + j);
      __syncwarp();
      if (t.up) {  // the first word without the elements before the staged part
        if (lane == 0) sw[0] &= ~0ull << (__ldg(t.vals + s0) & 63);
        __syncwarp();
      }
      st.words = sw;
      return P_SBITS;
    }
    if (zbits_words(a.n, len) <= (uint32_t)cap_words) {
      // compressed: 32 words per step, 4 steps of loads in flight
      const uint32_t groups = (a.n + 31) / 32;
      uint2* pz = reinterpret_cast<uint2*>(sm);
      uint64_t* zw = reinterpret_cast<uint64_t*>(sm + 2 * groups);
      const uint64_t* src = t.bs_words + a.off;
      uint32_t run = 0;
      for (uint32_t g0 = 0; g0 < groups; g0 += 4) {
        uint64_t x[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const uint32_t j = (g0 + u) * 32 + lane;
          x[u] = j < a.n ? __ldg(src + j) : 0ull;
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
          if (g0 + u < groups) {
            const uint32_t bal = __ballot_sync(kFull, x[u] != 0ull);
            if (x[u]) zw[run + __popc(bal & lanemask_lt())] = x[u];
            if (lane == 0) pz[g0 + u] = make_uint2(bal, run);
            run += __popc(bal);
          }
        }
      }
      __syncwarp();
      st.pz = pz;
      st.words = zw;
      return P_ZBITS;
    }
    st.words = t.bs_words + a.off;
    return P_GBITS;
  }
  if (layout == EH_LAYOUT_BLOCK_BITSET && !(blocks_too && len <= (uint32_t)cap_words)) {
    st.ids = t.bb_id + a.off;
    st.bwords = t.bb_words + 4 * a.off;
    st.n = a.n;
    return P_GBLOCK;
  }
  st.n = len;
  // A uint list staged in the triangle COUNT kernel becomes a compressed bitmap
  // (the P_ZBITS form, built from the sorted elements: presence bits by
  // shared atomics, ranks by a warp scan, each element's bit OR-ed into its
  // non-zero word) when that fits: two shared loads per probe in place of a
  // ~8-step binary search (R-MAT-22, density rule: 49.8 -> 28.7 warp-cycles
  // per probe including the build, kernel 9.91 -> 8.19 ms).
  if (zlist && len >= 2) {
    const uint32_t first = __ldg(t.vals + s0), last = __ldg(t.vals + s0 + len - 1);
    const uint32_t W = (last >> 6) - (first >> 6) + 1;
    // a plain bitmap, one load per probe, where it fits and clearing it is not
    // the larger part of building it (Chung-Lu 2^21, triangle: 3.87 -> 3.53 ms;
    // sets of a few elements over hundreds of words stay compressed)
    if (2 * W <= (uint32_t)cap_words && W <= 8 * len) {
      const uint32_t start = first >> 6;
      for (uint32_t j = lane; j < 2 * W; j += 32) sm[j] = 0u;
      __syncwarp();
      for (uint32_t j = lane; j < len; j += 32) {
        const uint32_t v = __ldg(t.vals + s0 + j);
        atomicOr(sm + ((v >> 5) - 2 * start), 1u << (v & 31));
      }
      __syncwarp();
      st.words = reinterpret_cast<uint64_t*>(sm);
      st.start = start;
      st.n = W;
      return P_SBITS;
    }
    if (zbits_words(W, len) <= (uint32_t)cap_words) {
      const uint32_t groups = (W + 31) / 32, start = first >> 6;
      uint2* pz = reinterpret_cast<uint2*>(sm);
      uint64_t* zw = reinterpret_cast<uint64_t*>(sm + 2 * groups);
      for (uint32_t g = lane; g < groups; g += 32) pz[g] = make_uint2(0u, 0u);
      __syncwarp();
      for (uint32_t j = lane; j < len; j += 32) {  // presence of each element's word
        const uint32_t k = (__ldg(t.vals + s0 + j) >> 6) - start;
        atomicOr(&pz[k >> 5].x, 1u << (k & 31));
      }
      __syncwarp();
      uint32_t run = 0;  // non-zero words before each group: a scan over the groups
      for (uint32_t g0 = 0; g0 < groups; g0 += 32) {
        const uint32_t g = g0 + lane;
        const uint32_t c = g < groups ? __popc(pz[g].x) : 0u;
        const uint32_t incl = warp_incl_scan(c);
        if (g < groups) pz[g].y = run + incl - c;
        run += __shfl_sync(kFull, incl, 31);
      }
      for (uint32_t j = lane; j < run; j += 32) zw[j] = 0ull;
      __syncwarp();
      for (uint32_t j = lane; j < len; j += 32) {  // each element's bit in its word
        const uint32_t v = __ldg(t.vals + s0 + j);
        const uint32_t k = (v >> 6) - start;
        const uint2 g = pz[k >> 5];
        atomicOr(reinterpret_cast<unsigned long long*>(zw + g.y + __popc(g.x & ((1u << (k & 31)) - 1u))),
                 1ull << (v & 63));
      }
      __syncwarp();
      st.pz = pz;
      st.words = zw;
      st.start = start;
      st.n = W;
      return P_ZBITS;
    }
  }
  if (len <= (uint32_t)cap_words) {
    for (uint32_t j = lane; j < len; j += 32) sm[j] = __ldg(t.vals + s0 + j);
    __syncwarp();
    st.list = sm;
    return P_SLIST;
  }
  st.list = t.vals + s0;
  return P_GLIST;
}

// One timing record of an item (eh_timing_records): warp-cycles spent on it
// beside the staged set's features.
__device__ __forceinline__ void write_record(float* rec, const TrieView& t, const RevView& r, const Item& item,
                                             int mode, float cycles) {
  const uint64_t b0 = t.off[item.hb];
  const uint32_t len = (uint32_t)(t.off[item.hb + 1] - b0);
  const uint32_t first = t.vals[b0], last = t.vals[b0 + len - 1];
  rec[0] = (float)len;
  rec[1] = (float)(r.rev_wpre[item.ke] - r.rev_wpre[item.kb]);
  rec[2] = (float)len / (float)(last - first + 1);
  rec[3] = (float)(last - first);
  rec[4] = (float)t.layout[item.hb];
  rec[5] = (float)mode;
  rec[6] = __uint_as_float(item.hb);  // set id, bit pattern
  rec[7] = cycles;
}

// stage_set for a block item: every thread of the block copies, into the
// block's whole shared region (the caller synchronises the block after).
__device__ __forceinline__ int stage_set_block(const TrieView& t, uint32_t hb, uint32_t* sm, int cap_words,
                                               Staged& st) {
  const uint8_t layout = t.layout[hb];
  const StagedRange sr = staged_range(t, hb);
  const uint64_t s0 = sr.s0;
  const uint32_t len = sr.len;
  const SetAux a = layout == EH_LAYOUT_RANGE_BITSET ? staged_bits(t, hb, sr) : t.aux[hb];
  if (layout == EH_LAYOUT_RANGE_BITSET) {
    st.start = a.start;
    st.n = a.n;
    if (2 * a.n <= (uint32_t)cap_words) {
      uint64_t* sw = reinterpret_cast<uint64_t*>(sm);
      for (uint32_t j = threadIdx.x; j < a.n; j += blockDim.x) {
        uint64_t w = __ldg(t.bs_words + a.off + j);
        if (t.up && j == 0) w &= ~0ull << (__ldg(t.vals + s0) & 63);  // as in stage_set
        sw[j] = w;
      }
      st.words = sw;
      return P_SBITS;
    }
    st.words = t.bs_words + a.off;
    return P_GBITS;
  }
  if (layout == EH_LAYOUT_BLOCK_BITSET) {
    st.ids = t.bb_id + a.off;
    st.bwords = t.bb_words + 4 * a.off;
    st.n = a.n;
    return P_GBLOCK;
  }
  st.n = len;
  if (len <= (uint32_t)cap_words) {
    for (uint32_t j = threadIdx.x; j < len; j += blockDim.x) sm[j] = __ldg(t.vals + s0 + j);
    st.list = sm;
    return P_SLIST;
  }
  st.list = t.vals + s0;
  return P_GLIST;
}

template <int kMode>
__device__ __forceinline__ uint64_t rows_of(int mode, const Staged& st, const TrieView& t, const RevView& r,
                                            uint32_t kb, uint32_t ke, uint32_t long_row, const Sink& sk) {
  if constexpr (kMode == MODE_COUNT) {
    switch (mode) {
      case P_SBITS: return count_rows<P_SBITS>(st, t, r, kb, ke, long_row);
      case P_GBITS: return count_rows<P_GBITS>(st, t, r, kb, ke, long_row);
      case P_SLIST: return count_rows<P_SLIST>(st, t, r, kb, ke, long_row);
      case P_GLIST: return count_rows<P_GLIST>(st, t, r, kb, ke, long_row);
      case P_ZBITS: return count_rows<P_ZBITS>(st, t, r, kb, ke, long_row);
      default: return count_rows<P_GBLOCK>(st, t, r, kb, ke, long_row);
    }
  } else {
    switch (mode) {
      case P_SBITS: return stream_rows<P_SBITS, kMode>(st, t, r, kb, ke, long_row, sk);
      case P_GBITS: return stream_rows<P_GBITS, kMode>(st, t, r, kb, ke, long_row, sk);
      case P_SLIST: return stream_rows<P_SLIST, kMode>(st, t, r, kb, ke, long_row, sk);
      case P_GLIST: return stream_rows<P_GLIST, kMode>(st, t, r, kb, ke, long_row, sk);
      case P_ZBITS: return stream_rows<P_ZBITS, kMode>(st, t, r, kb, ke, long_row, sk);
      default: return stream_rows<P_GBLOCK, kMode>(st, t, r, kb, ke, long_row, sk);
    }
  }
}

// A rank's part of the 4-clique of a relation that has an order (up, down,
// symmetric): the cliques whose lowest vertex (highest, going down) is head entry
// a belong to the rank of a.  A part so wide that, if it were dense, it would be
// more than an even share of the work (hits_work) is dealt out instead, eight rows
// a->b at a time by their position (eh_hits.cuh), and every rank makes its masks:
// one vertex next to most others would leave the other ranks idle (R-MAT-16 by its
// own ids in 8 shares: 30.9 ms on one rank, 1 to 6 on the others; so 6.1 to 7.0
// on each).  The rule asks the relation and
// the number of ranks alone, so that with or without masks the ranks cut alike.
struct CliqueShare {
  uint32_t index = 0, count = 1;
  uint32_t wide = 0xffffffffu;  // parts of at least this many elements are dealt out; above 32
  __device__ __forceinline__ bool builds(uint32_t a, uint32_t d) const {
    return count == 1 || d >= wide || a % count == index;
  }
  __device__ __forceinline__ bool owns(uint32_t a, uint32_t d, uint32_t i) const {
    return count == 1 || (d >= wide ? i >> 3 : a) % count == index;
  }
};

struct QueryOut {
  uint32_t long_row;                  // size-class boundary of rows (warp-wide vs flattened)
  unsigned long long* total;   // per graph results (one per trie)
  unsigned long long* annot;   // per head entry annotation or null
  float* records;              // per item timing records or null
  unsigned int* queue;         // [2] atomic queue heads: warp items, block items
  const unsigned int* n_items; // [2] warp items, block items
  const Item* bitems;          // MODE_COUNT: the block items
  unsigned long long* item_counts;  // per item count x count_mult (materialize sizing) or null
  uint32_t count_mult;
  const unsigned long long* item_off;  // MODE_MAT: first output row of each item
  uint32_t *ma, *mb, *mc;      // MODE_MAT: output columns
  const uint32_t* sel;         // 4-clique: bit per node value of a selected partner set, or null
  int32_t hot[kHot];           // MODE_ANNOT on a symmetric relation: largest sets' head entries, -1 if none
  uint32_t* gsbuf;             // 4-clique: per-warp S buffers in global memory (sets too large for
  uint32_t gcap;               //   shared memory), gcap words each; null: S in shared memory
  CliqueShare share;           // 4-clique without masks of an ordered relation: this rank's rows
};

// kOne: one trie, whose views are the kernel's parameters -- operands from the
// constant bank, where copies of a batch's views take two dozen registers.
template <int kMode, bool kOne>
__global__ void EH_TRI_LAUNCH_BOUNDS triangle_kernel(const __grid_constant__ TrieView t1,
                                                        const __grid_constant__ RevView r1,
                                                        const TrieView* __restrict__ views,
                                                        const RevView* __restrict__ revs,
                                                        const Item* __restrict__ items, int cap_words,
                                                        QueryOut out) {
  extern __shared__ uint32_t smem[];
  __shared__ unsigned int slot[kMaxWarps];  // MODE_MAT: rows written by the warp's item so far
  __shared__ unsigned long long hot_acc[kHot];
  __shared__ int32_t hot[kHot];
  if (kMode == MODE_ANNOT) {
    if (threadIdx.x < kHot) {
      hot_acc[threadIdx.x] = 0;
      hot[threadIdx.x] = out.hot[threadIdx.x];
    }
    __syncthreads();
  }
  const uint32_t lane = lane_id();
  const uint32_t wid = threadIdx.x >> 5;
  uint32_t* sm = smem + (size_t)wid * cap_words;
  unsigned long long acc = 0;
  uint32_t cur_g = 0xffffffffu;
  // Block items first (MODE_COUNT only): the block pulls an item, stages its
  // N(b) across the whole shared region, and its warps take the rows a few at a
  // time from a block counter.  Then each warp pulls warp items on its own.
  __shared__ unsigned int s_q, s_next;
  const uint32_t nwarps = blockDim.x >> 5;
  // a batch's current views, per warp: read where they are used instead of
  // held in two dozen registers
  __shared__ TrieView s_view[kOne ? 1 : kMaxWarps];
  __shared__ RevView s_rev[kOne ? 1 : kMaxWarps];
  uint32_t view_g = 0xffffffffu;
  const uint32_t n_witems = __ldg(out.n_items), n_bitems = kMode == MODE_COUNT ? __ldg(out.n_items + 1) : 0u;
  bool block_phase = n_bitems != 0;
  for (;;) {
    uint32_t it;
    if (block_phase) {
      if (threadIdx.x == 0) {
        s_q = atomicAdd(out.queue + 1, 1u);
        s_next = 0;
      }
      __syncthreads();
      it = s_q;
      if (it >= n_bitems) {  // the same on every thread of the block
        block_phase = false;
        continue;
      }
    } else {
      uint32_t q = 0;
      if (lane == 0) q = atomicAdd(out.queue, 1u);
      it = __shfl_sync(kFull, q, 0);
      if (it >= n_witems) break;
    }
    const Item item = block_phase ? out.bitems[it] : items[it];
    if (block_phase) it += n_witems;  // records: the warp items', then the block items'

    if (item.g != cur_g) {  // flush the running count of the previous graph
      if (lane == 0 && cur_g != 0xffffffffu && acc) atomicAdd(out.total + cur_g, acc);
      acc = 0;
      cur_g = item.g;
    }
    if (!kOne && item.g != view_g) {
      view_g = item.g;
      __syncwarp();
      if (lane == 0) {
        s_view[wid] = views[item.g];
        s_rev[wid] = revs[item.g];
      }
      __syncwarp();
    }
    const TrieView& t = kOne ? t1 : s_view[kOne ? 0 : wid];
    const RevView& r = kOne ? r1 : s_rev[kOne ? 0 : wid];
    long long t0 = 0;
    if (out.records && lane == 0) t0 = clock64();
    Sink sk{out.annot, out.ma, out.mb, out.mc, 0, &slot[wid], 0, hot, hot_acc, nullptr, 0, nullptr, nullptr,
            nullptr, 0, 0};
    if (kMode == MODE_MAT) {
      if (lane == 0) slot[wid] = 0;
      __syncwarp();
      sk.base = out.item_off[it];
      sk.b = t.head[item.hb];
    }
    Staged st;
    int mode;
    const bool merged = kMode == MODE_COUNT && (item.hb & kMerged);
    if (merged) {
      mode = P_GLIST;
    } else if (block_phase) {
      mode = stage_set_block(t, item.hb, smem, cap_words * (int)nwarps, st);
      __syncthreads();
    } else {
      // bitmaps for the annotation of an ordered or general relation too (kernel ms, star
      // of 2^16 leaves 5.4 -> 3.3, R-MAT-18 going down by degree 15.2 -> 7.0, R-MAT-20
      // 2.45 -> 2.0); a symmetric one's per-element counters are indexed by position in
      // the list
      const bool bitmap = kMode == MODE_COUNT ? !few_candidates(r, item)
                                              : kMode == MODE_ANNOT && r.dir != DIR_SYM && many_candidates(r, item);
      mode = stage_set(t, item.hb, sm, cap_words, st, bitmap);
    }
    const StagedRange sr = kMode == MODE_ANNOT ? staged_range(t, item.hb) : StagedRange{0, 0};
    const uint32_t blen = sr.len;
    if (kMode == MODE_ANNOT && r.dir == DIR_SYM && (mode == P_SLIST || mode == P_SBITS)) {
      // per-element counters after the staged structure, if they fit
      const uint32_t used = mode == P_SLIST ? st.n : 3 * st.n;  // list, or words (2 per) + ranks
      if (used + blen <= (uint32_t)cap_words) {
        sk.wmode = mode;
        sk.wn = st.n;
        sk.wlist = st.list;
        sk.wwords = st.words;
        sk.wstart = st.start;
        if (mode == P_SBITS) {
          uint32_t* rk = sm + 2 * st.n;
          // ranks within the staged part (none before its first word)
          const uint32_t* grk = t.bs_rank + staged_bits(t, item.hb, sr).off;
          const uint32_t before = (uint32_t)(sr.s0 - t.off[item.hb]);
          for (uint32_t j = lane; j < st.n; j += 32) rk[j] = j ? __ldg(grk + j) - before : 0u;
          sk.wrank = rk;
        }
        sk.wcnt = sm + used;
        for (uint32_t j = lane; j < blen; j += 32) sk.wcnt[j] = 0;
        __syncwarp();
      }
    }
    uint64_t c = 0;
    if (kMode == MODE_COUNT && merged) {
      c = count_merged(t, r, item.hb & ~kMerged, item.kb, item.ke);
    } else if (block_phase) {
      // rows at a time: 32, fewer where an item has few (and so long) rows, or one
      // warp takes them all (hubs among the low ids, kernel ms: Chung-Lu 2^18 by
      // descending degree 8.8 -> 7.8, R-MAT-18 going down by degree 7.3 -> 6.3)
      const uint32_t step = min(32u, max(1u, (item.ke - item.kb) / (4 * nwarps)));
      for (;;) {
        uint32_t batch = 0;
        if (lane == 0) batch = atomicAdd(&s_next, 1u);
        batch = __shfl_sync(kFull, batch, 0);
        const uint64_t k0 = (uint64_t)item.kb + (uint64_t)step * batch;
        if (k0 >= item.ke) break;
        const uint32_t k1 = k0 + step < (uint64_t)item.ke ? (uint32_t)(k0 + step) : item.ke;
        c += rows_of<kMode>(mode, st, t, r, (uint32_t)k0, k1, out.long_row, sk);
      }
    } else {
      c = rows_of<kMode>(mode, st, t, r, item.kb, item.ke, out.long_row, sk);
    }
    c = warp_sum(c);
    if (kMode == MODE_ANNOT && sk.wcnt) {  // flush the item's per-element counts
      __syncwarp();
      for (uint32_t j = lane; j < blen; j += 32) {
        const uint32_t n = sk.wcnt[j];
        if (n) atomicAdd(out.annot + __ldg(t.head_index + __ldg(t.vals + sr.s0 + j)), 2ull * n);
      }
    }
    if (kMode == MODE_ANNOT && r.dir == DIR_SYM && lane == 0 && c) atomicAdd(out.annot + item.hb, 2ull * c);
    if (out.item_counts && lane == 0) out.item_counts[it] = c * out.count_mult;
    acc += c;
    if (block_phase) __syncthreads();  // every warp is done with the staged set
    else __syncwarp();                 // the staged region is reused by the next item
    if (out.records && (block_phase ? threadIdx.x == 0 : lane == 0))
      write_record(out.records + 8 * (size_t)it, t, r, item, mode,
                   (float)(clock64() - t0) * (block_phase ? (float)nwarps : 1.f));  // warp-cycles
  }
  if (lane == 0 && cur_g != 0xffffffffu && acc) atomicAdd(out.total + cur_g, acc);
  if (kMode == MODE_ANNOT) {  // every warp leaves the loop above; then flush the block's hot counts
    __syncthreads();
    if (threadIdx.x < kHot && hot[threadIdx.x] >= 0 && hot_acc[threadIdx.x])
      atomicAdd(out.annot + hot[threadIdx.x], hot_acc[threadIdx.x]);
  }
}

// ------------------------------------------------------------ 4-clique
// For every row a->b: S = candidates(a,b) ∩ N(b) is materialised in the
// warp's shared region, then for each c in S the elements d of S are probed
// in N(c).  On an up- or down-oriented relation (or a symmetric one, rows
// a<b) only the d on the far side of c can close a 4-clique; on a general
// relation (self-loops, rows in both directions that are not symmetric) the
// candidates are the whole N(a) and every d of S is probed: the count is the
// number of assignments (a,b,c,d) with all six rows present, which is what
// the reference's N-way loop nest counts (TrieBuilder.cpp:276-348).
__device__ __forceinline__ uint32_t probe_global_set(const TrieView& t, uint32_t hc, uint32_t w) {
  const uint8_t layout = t.layout[hc];
  const SetAux a = t.aux[hc];
  if (layout == EH_LAYOUT_RANGE_BITSET) {
    Staged st;
    st.words = t.bs_words + a.off;
    st.start = a.start;
    st.n = a.n;
    return probe<P_GBITS>(st, w);
  }
  if (layout == EH_LAYOUT_BLOCK_BITSET) {
    Staged st;
    st.ids = t.bb_id + a.off;
    st.bwords = t.bb_words + 4 * a.off;
    st.n = a.n;
    return probe<P_GBLOCK>(st, w);
  }
  const uint64_t s0 = t.off[hc];
  const uint32_t n = (uint32_t)(t.off[hc + 1] - s0);
  if (!n) return 0;
  return list_contains<false>(t.vals + s0, n, w) ? 1u : 0u;
}

__device__ __forceinline__ uint32_t sel_bit(const uint32_t* sel, uint32_t x) {
  return (__ldg(sel + (x >> 5)) >> (x & 31)) & 1u;
}

// With a selection (sel != null, bit per node value of the partner set
// {a : (a,v) in Edge}), only 4-cliques whose root a is selected count.  On
// an oriented relation the row's a is the plan's root: other rows are
// skipped.  On a symmetric relation the one undirected clique found stands
// for its 4! orderings, of which 3! start at each member: the hit counts
// the members that are selected (the host multiplies by 3!).
template <int P>
__device__ uint64_t clique_rows(const Staged& st, const TrieView& t, const RevView& r, uint32_t kb, uint32_t ke,
                                uint32_t* sbuf, uint32_t cap, const uint32_t* sel, uint32_t wb,
                                const CliqueShare& share) {
  const uint32_t lane = lane_id();
  const bool up = r.dir != DIR_DOWN;
  const bool general = r.dir == DIR_GENERAL;
  uint64_t cnt = 0;
  for (uint32_t k = kb; k < ke; k++) {
    uint32_t wab = 0;
    if (sel) {
      const uint32_t wa = sel_bit(sel, __ldg(t.head + __ldg(r.rev_src + k)));
      if (r.dir != DIR_SYM && !wa) continue;  // warp-uniform: k is the same on every lane
      wab = wa + wb;
    }
    const uint32_t lo = __ldg(r.rev_lo + k), hi = __ldg(r.rev_hi + k);
    if (share.count > 1) {
      const uint32_t a = __ldg(r.rev_src + k), d = staged_range(t, a).len;
      if (!share.owns(a, d, d - 1 - (hi - lo))) continue;
    }
    // S = N(a)[lo, hi) ∩ N(b), compacted in order
    uint32_t ns = 0;
    for (uint32_t base = lo; base < hi; base += 32) {
      const uint32_t e = base + lane;
      uint32_t w = 0, hit = 0;
      if (e < hi) {
        w = __ldg(t.vals + e);
        hit = probe<P>(st, w);
      }
      const uint32_t ball = __ballot_sync(kFull, hit);
      if (hit) {
        const uint32_t pos = ns + __popc(ball & lanemask_lt());
        if (pos < cap) sbuf[pos] = w;
      }
      ns += __popc(ball);
    }
    __syncwarp();
    if (ns > cap) ns = cap;  // capacity bound checked by the host planner
    // small S: the (c, d) pairs flattened over the lanes, so a warp step
    // probes 32 pairs whatever the length of each c's run
    if (ns <= kFlatClique) {
      const uint32_t np = general ? ns * ns : ns * (ns - 1) / 2;
      for (uint32_t p = lane; p < np; p += 32) {
        uint32_t i, j;  // the pair's positions in S: i < j unless general
        if (general) {
          i = p / ns;
          j = p - i * ns;
        } else {
          // row i of the triangular pair index holds ns - 1 - i pairs and
          // starts at i * ns - i * (i + 1) / 2; a float guess, then exact steps
          const float m = (float)(2 * ns - 1);
          int g = (int)floorf((m - sqrtf(fmaxf(m * m - 8.f * (float)p, 0.f))) * 0.5f);
          g = max(0, min(g, (int)ns - 2));
          i = (uint32_t)g;
          while (i + 1 < ns - 1 && (i + 1) * ns - (i + 1) * (i + 2) / 2 <= p) i++;
          while (i > 0 && i * ns - i * (i + 1) / 2 > p) i--;
          j = p - (i * ns - i * (i + 1) / 2) + i + 1;
        }
        // up (and general): probe d = S[j] in N(S[i]); down: d = S[i] in N(S[j])
        const uint32_t c = (up || general) ? sbuf[i] : sbuf[j];
        const uint32_t dd = (up || general) ? sbuf[j] : sbuf[i];
        const int32_t hc = __ldg(t.head_index + c);
        if (hc < 0) continue;
        if (probe_global_set(t, (uint32_t)hc, dd))
          cnt += (sel && r.dir == DIR_SYM) ? wab + sel_bit(sel, c) + sel_bit(sel, dd) : 1u;
      }
      __syncwarp();
      continue;
    }
    // for each c = S[i]: count S elements beyond c (up) or before c (down) in N(c)
    for (uint32_t i = 0; i < ns; i++) {
      const uint32_t c = sbuf[i];
      const int32_t hc = __ldg(t.head_index + c);
      if (hc < 0) continue;
      const uint32_t jb = general ? 0 : (up ? i + 1 : 0), je = general ? ns : (up ? ns : i);
      if (sel && r.dir == DIR_SYM) {
        const uint32_t wabc = wab + sel_bit(sel, c);
        for (uint32_t j = jb + lane; j < je; j += 32)
          if (probe_global_set(t, (uint32_t)hc, sbuf[j])) cnt += wabc + sel_bit(sel, sbuf[j]);
      } else {
        for (uint32_t j = jb + lane; j < je; j += 32) cnt += probe_global_set(t, (uint32_t)hc, sbuf[j]);
      }
    }
    __syncwarp();
  }
  return cnt;
}

__global__ void EH_TRI_LAUNCH_BOUNDS clique4_kernel(const TrieView* __restrict__ views,
                                                       const RevView* __restrict__ revs,
                                                       const Item* __restrict__ items, int cap_words,
                                                       QueryOut out) {
  extern __shared__ uint32_t smem[];
  const uint32_t lane = lane_id();
  const uint32_t wid = threadIdx.x >> 5;
  uint32_t* sm = smem + (size_t)wid * cap_words;
  // S after the staged set in the warp's region, or in its global buffer
  const int half = out.gsbuf ? cap_words : cap_words / 2;
  uint32_t* sbuf = out.gsbuf ? out.gsbuf + ((size_t)blockIdx.x * (blockDim.x >> 5) + wid) * out.gcap : sm + half;
  const uint32_t scap = out.gsbuf ? out.gcap : (uint32_t)half;
  unsigned long long acc = 0;
  uint32_t cur_g = 0xffffffffu;
  const uint32_t n_items = __ldg(out.n_items);
  for (;;) {
    uint32_t it = 0;
    if (lane == 0) it = atomicAdd(out.queue, 1u);
    it = __shfl_sync(kFull, it, 0);
    if (it >= n_items) break;
    const Item item = items[it];
    if (item.g != cur_g) {
      if (lane == 0 && cur_g != 0xffffffffu && acc) atomicAdd(out.total + cur_g, acc);
      acc = 0;
      cur_g = item.g;
    }
    const TrieView t = views[item.g];
    const RevView r = revs[item.g];
    long long t0 = 0;
    if (out.records && lane == 0) t0 = clock64();
    Staged st;
    const int mode = stage_set(t, item.hb, sm, half, st);
    const uint32_t wb = out.sel ? sel_bit(out.sel, t.head[item.hb]) : 0u;
    uint64_t c;
    switch (mode) {
      case P_SBITS: c = clique_rows<P_SBITS>(st, t, r, item.kb, item.ke, sbuf, scap, out.sel, wb, out.share); break;
      case P_GBITS: c = clique_rows<P_GBITS>(st, t, r, item.kb, item.ke, sbuf, scap, out.sel, wb, out.share); break;
      case P_SLIST: c = clique_rows<P_SLIST>(st, t, r, item.kb, item.ke, sbuf, scap, out.sel, wb, out.share); break;
      case P_GLIST: c = clique_rows<P_GLIST>(st, t, r, item.kb, item.ke, sbuf, scap, out.sel, wb, out.share); break;
      case P_ZBITS: c = clique_rows<P_ZBITS>(st, t, r, item.kb, item.ke, sbuf, scap, out.sel, wb, out.share); break;
      default: c = clique_rows<P_GBLOCK>(st, t, r, item.kb, item.ke, sbuf, scap, out.sel, wb, out.share); break;
    }
    acc += warp_sum(c);
    __syncwarp();
    if (out.records && lane == 0)
      write_record(out.records + 8 * (size_t)it, t, r, item, mode, (float)(clock64() - t0));
  }
  if (lane == 0 && cur_g != 0xffffffffu && acc) atomicAdd(out.total + cur_g, acc);
}

}  // namespace eh

#include "eh_hits.cuh"

namespace eh {

// ------------------------------------------------- lollipop / barbell roots
constexpr uint64_t kRootBig = 4096;  // barbell root: larger sets are shared by the whole grid

// LollipopAgg root, order [a,d]: sum_a T(a) * |N(a)|
// BarbellAgg root, order [a,x]: sum_a T(a) * sum_{x in N(a) ∩ head} T(x);
// Tv = T by value (0 off the head): one random load per row instead of two.
// A warp per set: a hub's 32 K elements in one warp took 0.53 ms of the 1.27
// of a barbell on 2^16 nodes, so larger sets are left to root_big_kernel; and on
// a symmetric relation the sum over rows (a,x) of T(a) T(x) is twice that over
// the rows a < x.
template <bool kBarbell>
__global__ void root_kernel(TrieView t, const unsigned long long* __restrict__ T,
                            const unsigned long long* __restrict__ Tv, unsigned long long* __restrict__ total,
                            uint32_t* __restrict__ big, unsigned int* __restrict__ n_big) {
  const uint32_t lane = lane_id();
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  unsigned long long acc = 0;
  if (!kBarbell) {
    for (uint32_t a = blockIdx.x * blockDim.x + threadIdx.x; a < t.n_head; a += gridDim.x * blockDim.x)
      acc += T[a] * (t.off[a + 1] - t.off[a]);
    acc = warp_sum(acc);
  } else {
    for (uint32_t a = warp; a < t.n_head; a += nwarps) {
      const unsigned long long ta = T[a];
      if (!ta) continue;
      const StagedRange r = staged_range(t, a);
      if (r.len > kRootBig) {
        if (lane == 0) big[atomicAdd(n_big, 1u)] = a;
        continue;
      }
      unsigned long long s = 0;
      for (uint32_t e = lane; e < r.len; e += 32) s += __ldg(Tv + __ldg(t.vals + r.s0 + e));
      acc += ta * s;
    }
    acc = warp_sum(acc) * (t.up ? 2ull : 1ull);
  }
  if (lane == 0 && acc) atomicAdd(total, acc);
}

// the barbell root of the large sets, each grid-wide
__global__ void root_big_kernel(TrieView t, const uint32_t* __restrict__ big, const unsigned int* __restrict__ n_big,
                                const unsigned long long* __restrict__ T, const unsigned long long* __restrict__ Tv,
                                unsigned long long* __restrict__ total) {
  unsigned long long acc = 0;
  const unsigned int n = *n_big;
  for (unsigned int k = 0; k < n; k++) {
    const uint32_t a = big[k];
    const StagedRange r = staged_range(t, a);
    unsigned long long s = 0;
    for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < r.len; e += (uint64_t)gridDim.x * blockDim.x)
      s += __ldg(Tv + __ldg(t.vals + r.s0 + e));
    acc += T[a] * s;
  }
  acc = warp_sum(acc) * (t.up ? 2ull : 1ull);
  if (lane_id() == 0 && acc) atomicAdd(total, acc);
}

__global__ void t_by_value_kernel(TrieView t, const unsigned long long* __restrict__ T,
                                  unsigned long long* __restrict__ Tv) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < t.n_nodes; v += gridDim.x * blockDim.x) {
    const int32_t h = t.head_index[v];
    Tv[v] = h >= 0 ? T[h] : 0ull;
  }
}

// ---------------------------------------------------------------- driver
static RevView rev_view(const eh_trie* t) {
  return RevView{t->rev_off.p, t->rev_lo.p, t->rev_hi.p, t->rev_src.p, t->rev_wpre.p, t->dir};
}

// What a kernel may use and how many of its blocks an SM holds are constants of
// the device: asked of the runtime once per kernel (and launch shape), not on
// every query (some 8 us of a small one).  A kernel's dynamic shared memory limit
// is raised to all it may use the first time.
struct KernelShapes {
  std::mutex mu;
  struct Room {
    const void* kernel;
    int device;
    size_t bytes;
  };
  struct Blocks {
    const void* kernel;
    int device, threads;
    size_t smem;
    int blocks;
  };
  std::vector<Room> rooms;
  std::vector<Blocks> blocks;
};
static KernelShapes& kernel_shapes() {
  static KernelShapes k;
  return k;
}

// dynamic shared memory a block of `kernel` may use: the device's opt-in
// per-block limit less the kernel's own static shared memory
static size_t dynamic_smem_room(const void* kernel) {
  int dev = 0, optin = 0;
  EH_CUDA(cudaGetDevice(&dev));
  KernelShapes& k = kernel_shapes();
  std::lock_guard<std::mutex> l(k.mu);
  for (const auto& r : k.rooms)
    if (r.kernel == kernel && r.device == dev) return r.bytes;
  EH_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  cudaFuncAttributes fa;
  EH_CUDA(cudaFuncGetAttributes(&fa, kernel));
  const size_t room = (size_t)optin > fa.sharedSizeBytes ? (size_t)optin - fa.sharedSizeBytes : 0;
  EH_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)room));
  k.rooms.push_back({kernel, dev, room});
  return room;
}
// after dynamic_smem_room(kernel)
static int blocks_per_sm(const void* kernel, int threads, size_t smem) {
  int dev = 0, b = 0;
  EH_CUDA(cudaGetDevice(&dev));
  KernelShapes& k = kernel_shapes();
  std::lock_guard<std::mutex> l(k.mu);
  for (const auto& x : k.blocks)
    if (x.kernel == kernel && x.device == dev && x.threads == threads && x.smem == smem) return x.blocks;
  EH_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, threads, smem));
  b = std::max(1, b);
  // 4-cliques without masks size their staging by the largest set: the oldest shapes go
  if (k.blocks.size() >= 64) k.blocks.erase(k.blocks.begin());
  k.blocks.push_back({kernel, dev, threads, smem, b});
  return b;
}

// Small device and pinned host memory of a context, kept from call to call (a
// caller holds the context's lock until its work is done): a query's plan and
// control block.  Past kMaxWorkspace a call allocates and frees its own.  Not in
// the stream-ordered pool: what a call took there goes back with it.
constexpr size_t kMaxWorkspace = 64ull << 20;
unsigned char* workspace(eh_context* ctx, size_t bytes) {
  if (bytes > kMaxWorkspace) return nullptr;
  if (bytes > ctx->work_cap) {
    EH_CUDA(cudaStreamSynchronize(ctx->stream));
    const size_t want = std::min(kMaxWorkspace, std::max<size_t>(bytes + bytes / 2, 1u << 20));
    void* p = nullptr;
    if (cudaMalloc(&p, want) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    if (ctx->work) cudaFree(ctx->work);
    ctx->work = (unsigned char*)p;
    ctx->work_cap = want;
  }
  return ctx->work;
}
unsigned char* pinned(eh_context* ctx, size_t bytes) {
  if (bytes > ctx->pinned_cap) {
    EH_CUDA(cudaStreamSynchronize(ctx->stream));
    if (ctx->pinned) EH_CUDA(cudaFreeHost(ctx->pinned));
    ctx->pinned = nullptr;
    ctx->pinned_cap = 0;
    EH_CUDA(cudaMallocHost((void**)&ctx->pinned, 2 * bytes + 4096));
    ctx->pinned_cap = 2 * bytes + 4096;
  }
  return ctx->pinned;
}

struct Launch {
  uint32_t launches = 0;
};

// The hit masks of a prepared launch (eh_hits.cuh): where every head entry's
// matrix and its second-pass units start, and the mask words.
struct Hits {
  bool on = false;
  int use = 0;
  uint64_t words = 0;
  uint32_t units = 0, heads = 0, n = 0;
  uint32_t longest = 0;   // longest part
  uint32_t launches = 0;  // kernels of the mask plan
  CliqueShare share;      // HITS_CLIQUE
  DevBuf<uint32_t> mask;
  DevBuf<uint32_t> plan;  // [heads] mask offsets, [heads + 1] units before, [n + 1] graph starts, sums
  DevBuf<uint32_t> heavy; // 4-clique with wide parts: HeavyUnits, the two counters first
  uint32_t* moff() const { return plan.p; }
  uint32_t* upre() const { return plan.p + heads; }
  uint32_t* gstart() const { return upre() + heads + 1; }
  HitsView view() const { return HitsView{mask.p, moff(), upre(), gstart(), n, heads, share}; }
};
// Masks hold a bit per candidate, so a relation in degree order needs far less
// than its trie (R-MAT-22: 1.2 GB); past this many words (8 GB: a set of 300 K
// elements read whole) the plans run without them.
constexpr uint64_t kMaxHitWords = 1ull << 31;
// Every rank that shares a 4-clique makes the masks of the widest parts (CliqueShare).
// Where the widest is so wide that the relation's rows can fill no more than a
// kSparseHub-th of its matrix, making it is nearly all of the query, and the plan
// without masks splits better (slowest of 8 shares, without / with, ms: star of 2^16
// leaves with 2^18 rows among them, filled to a 6500th at most, 1.3 / 3.4; of 2^13,
// an 800th, 0.23 / 0.27; R-MAT-16 by its own ids, a 50th, 134 / 7.6).
constexpr double kSparseHub = 1024;

// parts from this length on have more than a count-th of all the 4-clique's work
static uint32_t wide_part(uint64_t work, uint32_t longest, uint32_t count) {
  uint32_t lo = 33, hi = std::max(33u, longest + 1);
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo) / 2;
    if ((double)hits_work(mid) * count > (double)work) hi = mid; else lo = mid + 1;
  }
  return lo;
}

// Sizes and allocates the masks.  H.on: they are there.  H.share: how ranks share
// a 4-clique of this relation, with its masks or (no memory for them) without; of
// one rank (they share by items) if the relation is general, its masks are too large
// for any or not worth it for ranks, or no row has candidates: all facts of the
// relation, the same on every rank.
static void plan_hits(eh_context* ctx, const eh_trie* const* tries, uint32_t n, int use, const ExecParams& ep,
                      Hits& H) {
  cudaStream_t s = ctx->stream;
  uint64_t heads = 0, entries = 0, rows = 0;
  std::vector<uint32_t> gstart(n + 1, 0);
  for (uint32_t g = 0; g < n; g++) {
    const int dir = tries[g]->dir;
    if (dir == DIR_GENERAL || (use == HITS_ANNOT && dir != DIR_SYM) || (use == HITS_ROWS && dir == DIR_SYM)) return;
    heads += tries[g]->n_head;
    entries += tries[g]->rev_entries;
    rows += tries[g]->rows;
    if (heads >= (1ull << 32) - 1) return;
    gstart[g + 1] = (uint32_t)heads;
  }
  if (!entries) return;
  H.use = use;
  H.n = n;
  H.heads = (uint32_t)heads;
  const size_t o_sums = (2 * heads + 1 + n + 1 + 1) & ~(size_t)1;  // 64-bit sums
  H.plan.alloc(o_sums + 12, s);
  unsigned long long* sums = reinterpret_cast<unsigned long long*>(H.plan.p + o_sums);
  EH_CUDA(cudaMemsetAsync(H.upre() + heads, 0, 4, s));
  EH_CUDA(cudaMemcpyAsync(H.gstart(), gstart.data(), (n + 1) * 4, cudaMemcpyHostToDevice, s));
  // mask words, units and longest part of all head entries, bound of the 4-clique's work on them; words and
  // units of the head entries that `share` builds
  unsigned long long h[6];
  auto size = [&](const CliqueShare& share) {
    EH_CUDA(cudaMemsetAsync(sums, 0, sizeof(h), s));
    for (uint32_t g = 0; g < n; g++) {
      const uint32_t nh = tries[g]->n_head;
      if (!nh) continue;
      const int grid = std::min(num_sms() * 4, ceil_div(nh, 256));
      hits_size_kernel<<<grid, 256, 0, s>>>(tries[g]->view(), use, share, H.moff() + gstart[g], H.upre() + gstart[g],
                                            sums);
      EH_CHECK_LAUNCH();
      H.launches++;
    }
    EH_CUDA(cudaMemcpyAsync(h, sums, sizeof(h), cudaMemcpyDeviceToHost, s));
    EH_CUDA(cudaStreamSynchronize(s));
  };
  const bool shared = use == HITS_CLIQUE && ep.shard_count > 1;
  size(shared ? CliqueShare{ep.shard_index, ep.shard_count} : CliqueShare{});
  if (h[0] > kMaxHitWords || h[1] >= kMaxHitWords) return;
  H.longest = (uint32_t)h[2];
  if (shared && 0.5 * H.longest * H.longest > kSparseHub * rows) return;
  if (shared) {
    H.share = CliqueShare{ep.shard_index, ep.shard_count, wide_part(h[3], H.longest, ep.shard_count)};
    if (H.longest >= H.share.wide) size(H.share);  // once more with the wide ones
  }
  if (!ep.masks) return;
  exclusive_scan<uint32_t>(H.moff(), H.moff(), heads, nullptr, s);
  exclusive_scan<uint32_t>(H.upre(), H.upre(), heads + 1, nullptr, s);
  H.launches += scan_launches(heads) + scan_launches(heads + 1);
  try {
    H.mask.alloc(h[4] ? h[4] : 1, s);
    // a wide part has 4 (W + 1) mask words per unit
    if (use == HITS_CLIQUE && H.longest > 32 * kSparseWords)
      H.heavy.alloc(2 + std::min<uint64_t>(h[5], h[4] / (4 * kSparseWords)) + 1, s);
  } catch (const Error& e) {
    if (e.code != EH_ERR_OOM) throw;
    H.mask.release();
    return;
  }
  H.words = h[4];
  H.units = (uint32_t)h[5];
  H.on = true;
  if (ep.held) *ep.held = true;
}

// Masks are up to 8 GB.  A call that has them and then finds no memory for the rest
// of what it needs (a fine plan, materialized rows) gives them back and runs once
// more without: f(ExecParams) is the whole call, and holds its memory itself.
template <typename F>
static void with_or_without_masks(eh_context* ctx, ExecParams ep, F f) {
  bool held = false;
  ep.held = &held;
  try {
    f(ep);
    return;
  } catch (const Error& e) {
    if (e.code != EH_ERR_OOM || !held) throw;
  }
  EH_CUDA(cudaStreamSynchronize(ctx->stream));  // the first try's work; pinned memory is written again
  ep.masks = false;
  f(ep);
}

// Runs the intersection kernel of `query` over the concatenated plans of
// n graphs; results accumulate into d_total[g].
// Everything a launch needs on the device, built once: the work plans of
// the tries concatenated into one queue, their views, the launch shape.
struct Prepared {
  DevBuf<unsigned char> own;      // device arrays of a launch that outlives the call (a batch) or is large
  Control* ctl = nullptr;         // control block, results, views, items: one piece of device memory
  unsigned long long* total = nullptr;  // [n] results
  TrieView view0{};               // the first trie's views
  RevView rev0{};
  TrieView* dv = nullptr;
  RevView* dr = nullptr;
  Item* items = nullptr;          // warp items, at most cap_w
  Item* bitems = nullptr;         // block items, at most cap_b
  uint64_t cap_w = 0, cap_b = 0;
  uint32_t n = 0;                 // tries
  uint64_t entries = 0;           // rows of the tries' reverse levels: 0 means nothing to run
  uint64_t pairs = 0;
  ExecParams ep{};
  size_t smem = 0;
  int grid = 1, threads = 32;
  int query = 0;
  bool annot = false;
  uint32_t plan_launches = 0;
  const uint32_t* sel = nullptr;  // 4-clique selection bitmap (QueryOut::sel)
  DevBuf<uint32_t> gs;            // 4-clique global S buffers (ExecParams::s_cap)
  int32_t hot[kHot] = {-1, -1, -1, -1};  // annotation: largest sets (QueryOut::hot)
  Hits hits;                      // the plan runs on hit masks
  size_t ctl_bytes() const { return sizeof(Control) + n * sizeof(unsigned long long); }  // what comes back
};

// head entry with the largest set, excluding `ex` (-1 unused): max over
// (size << 32 | position)
__global__ void top_set_kernel(const uint64_t* __restrict__ off, uint32_t nh, Int4 ex,
                               unsigned long long* __restrict__ best) {
  unsigned long long m = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nh; i += gridDim.x * blockDim.x) {
    if ((int32_t)i == ex.v[0] || (int32_t)i == ex.v[1] || (int32_t)i == ex.v[2] || (int32_t)i == ex.v[3]) continue;
    m = max(m, (unsigned long long)(((off[i + 1] - off[i]) << 32) | i));
  }
  for (int o = 16; o; o >>= 1) m = max(m, __shfl_xor_sync(kFull, m, o));
  if (lane_id() == 0 && m) atomicMax(best, m);
}

// the kHot head entries with the largest sets of a trie (-1 where fewer); the
// kernels launched
static uint32_t hot_sets(eh_context* ctx, const eh_trie* t, int32_t* hot) {
  cudaStream_t s = ctx->stream;
  Int4 ex{{-1, -1, -1, -1}};
  DevBuf<unsigned long long> best(1, s);
  uint32_t launches = 0;
  for (int k = 0; k < kHot; k++) hot[k] = -1;
  for (int k = 0; k < kHot && (uint32_t)k < t->n_head; k++) {
    EH_CUDA(cudaMemsetAsync(best.p, 0, 8, s));
    top_set_kernel<<<num_sms() * 4, 256, 0, s>>>(t->off.p, t->n_head, ex, best.p);
    EH_CHECK_LAUNCH();
    launches++;
    unsigned long long h = 0;
    EH_CUDA(cudaMemcpyAsync(&h, best.p, 8, cudaMemcpyDeviceToHost, s));
    EH_CUDA(cudaStreamSynchronize(s));
    if (!h) break;
    hot[k] = (int32_t)(h & 0xffffffffu);
    ex.v[k] = hot[k];
  }
  return launches;
}

// 4-clique without hit masks: the warp's shared region holds the staged N(b) and S
// (S <= the largest set) while that stays within 96 KB a block; beyond, S
// moves to per-warp global buffers (L2-resident in practice) and the whole
// region stages N(b).
static void size_clique_staging(ExecParams& ep, uint32_t max_set) {
  const int need = 2 * ((int)max_set + 1);
  if ((size_t)std::max(ep.smem_words, need) * 4 * ep.warps <= 96 * 1024) {
    if (ep.smem_words < need) ep.smem_words = (need + 1) & ~1;
  } else {
    ep.s_cap = max_set + 1;
  }
}

// hits_use: run the plan on hit masks when they can be had (HITS_*; -1: never).
// keep: the launch outlives the call, so its device memory is its own.  merge:
// entries with little work may share items.
static void prepare(eh_context* ctx, const eh_trie* const* tries, uint32_t n, int query, ExecParams ep, bool annot,
                    Prepared& P, bool block_items = false, int hits_use = -1, bool keep = false,
                    bool merge = true) {
  cudaStream_t s = ctx->stream;
  P.query = query;
  P.annot = annot;
  if (hits_use >= 0) plan_hits(ctx, tries, n, hits_use, ep, P.hits);
  P.plan_launches += P.hits.launches;
  const bool hits = P.hits.on;
  if (hits_use == HITS_ROWS && !hits) return;  // rows come from masks, or from a plan made for them
  if (query == EH_QUERY_CLIQUE4 && !hits) {
    uint32_t mx = 0;
    for (uint32_t g = 0; g < n; g++) mx = std::max(mx, tries[g]->info.max_set);
    size_clique_staging(ep, mx);
  }
  // the launch shape first: the plan's classes depend on the staging capacity
  // the annotated pass of a symmetric relation stages more of N(b) by default: its
  // matched elements then count in shared memory (measured on Chung-Lu 2^23: 2048
  // words per warp 234 ms, 1024 245 ms)
  bool sym = false;
  for (uint32_t g = 0; g < n; g++) sym |= tries[g]->dir == DIR_SYM;
  if (annot && sym && !hits && !ep.smem_given) ep.smem_words = 2048;
  P.threads = 32 * ep.warps;
  P.smem = (size_t)ep.smem_words * 4 * ep.warps;
  const void* kfn;
  if (hits) kfn = n == 1 ? (const void*)hits_kernel<true> : (const void*)hits_kernel<false>;
  else if (query == EH_QUERY_CLIQUE4) kfn = (const void*)clique4_kernel;
  else if (annot) kfn = (const void*)triangle_kernel<MODE_ANNOT, true>;
  else kfn = n == 1 ? (const void*)triangle_kernel<MODE_COUNT, true> : (const void*)triangle_kernel<MODE_COUNT, false>;
  {
    size_t room = dynamic_smem_room(kfn);
    // the materializing pass launches MODE_MAT with the same shape
    if (!hits && !annot && query != EH_QUERY_CLIQUE4)
      room = std::min(room, dynamic_smem_room((const void*)triangle_kernel<MODE_MAT, true>));
    if (P.smem > room) {
      // shrink the per-warp region to what a block may hold (a staged set
      // that no longer fits is probed in global memory instead)
      EH_REQUIRE(query != EH_QUERY_CLIQUE4, EH_ERR_UNSUPPORTED, "4-clique staging exceeds shared memory");
      ep.smem_words = (int)((room / 4 / ep.warps) & ~(size_t)1);
      P.smem = (size_t)ep.smem_words * 4 * ep.warps;
    }
  }
  const int per_sm = blocks_per_sm(kfn, P.threads, P.smem);
  // block items only for the plain triangle COUNT
  const bool blocks_query = query == EH_QUERY_TRIANGLE && !annot;
  const bool blocks = block_items && !hits && query == EH_QUERY_TRIANGLE && !annot && ep.warps > 1 &&
                      !ep.no_block_items;
  // work of all tries, and how finely to cut it: 8 items for each resident
  // warp (of every rank), of kMinChunk to kMaxChunk at most
  uint64_t cost = 0, head_items = 0;
  P.n = n;
  for (uint32_t g = 0; g < n; g++) {
    P.entries += tries[g]->rev_entries;
    P.pairs += tries[g]->rev_pairs;
    cost += tries[g]->rev_pairs + kRowCost * tries[g]->rev_entries;
    head_items += std::min<uint64_t>(tries[g]->n_head, tries[g]->rev_entries);
  }
  // ranks that share a query cut the same items, whatever they run on
  const uint64_t resident = (uint64_t)num_sms() * per_sm * ep.warps;
  const uint64_t slots = ep.shard_count > 1 ? (uint64_t)kShareWarps * ep.shard_count : resident;
  if (!ep.chunk_given) {
    // a 4-clique without masks does far more per row than the plan weighs (selection
    // on R-MAT-18 going down by degree 548 ms; cut up to kMaxChunk 902), an annotation
    // without masks somewhat more
    const uint64_t most = (query == EH_QUERY_CLIQUE4 || annot) && !hits ? kDefaultChunk : kMaxChunk;
    ep.chunk = (uint32_t)std::min<uint64_t>(most, std::max<uint64_t>(kMinChunk, cost / (8 * slots)));
  }
  PlanShape shape{ep.chunk, nullptr, 0.0, (uint32_t)ep.smem_words,
                   blocks ? (uint32_t)ep.smem_words * (uint32_t)ep.warps : 0u, (uint32_t)ep.warps, 0u};
  // items: at most one per entry with rows and one per chunk of work; with predicted
  // costs one per chunk of predicted cycles (the sum of rounded-up shares; the slack
  // covers their rounding) and one per kPredTrust chunks of work
  bool pred = false;
  for (uint32_t g = 0; g < n; g++) pred |= tries[g]->work_pred.p != nullptr;
  const uint64_t chunks = cost / ep.chunk + (pred ? cost / (kPredTrust * ep.chunk) : 0);
  P.cap_w = head_items + chunks + chunks / 64 + 64;
  P.cap_b = blocks ? std::min<uint64_t>(P.cap_w, chunks / ep.warps + cost / kMinBlockWork + chunks / 64 + 64) : 0;
  EH_REQUIRE(P.cap_w < (1ull << 32), EH_ERR_UNSUPPORTED, "work plan of 2^32 items or more");
  const size_t o_views = (P.ctl_bytes() + 127) & ~(size_t)127;
  const size_t o_rev = o_views + n * sizeof(TrieView);
  const size_t head_bytes = o_rev + n * sizeof(RevView);
  uint32_t max_heads = 0;
  for (uint32_t g = 0; g < n; g++) max_heads = std::max(max_heads, tries[g]->n_head);
  const size_t o_pos = (head_bytes + 255) & ~(size_t)255;  // the planner's places and tile sums, trie by trie
  const size_t o_items = o_pos + (((size_t)max_heads + max_heads / kPlanTile + 1) * 8 + 255 & ~(size_t)255);
  const size_t bytes = o_items + (P.cap_w + P.cap_b) * sizeof(Item);
  unsigned char* base = keep ? nullptr : workspace(ctx, bytes);
  if (!base) {
    P.own.alloc(bytes, s);
    base = P.own.p;
  }
  P.ctl = reinterpret_cast<Control*>(base);
  P.total = reinterpret_cast<unsigned long long*>(base + sizeof(Control));
  P.dv = reinterpret_cast<TrieView*>(base + o_views);
  P.dr = reinterpret_cast<RevView*>(base + o_rev);
  P.items = reinterpret_cast<Item*>(base + o_items);
  P.bitems = P.items + P.cap_w;
  unsigned char* host = pinned(ctx, head_bytes);  // the last user of it has been waited for
  memset(host, 0, o_views);
  for (uint32_t g = 0; g < n; g++) {
    const TrieView v = tries[g]->view();
    const RevView r = rev_view(tries[g]);
    memcpy(host + o_views + g * sizeof(TrieView), &v, sizeof(v));
    memcpy(host + o_rev + g * sizeof(RevView), &r, sizeof(r));
    // the intersection kernels read the values and the bitset words with
    // 16-byte loads at 16-byte aligned indices
    if ((reinterpret_cast<uintptr_t>(v.vals) | reinterpret_cast<uintptr_t>(v.bs_words)) & 15u)
      throw Error{EH_ERR_UNSUPPORTED, "trie arrays are not 16-byte aligned"};
    if (!g) {
      P.view0 = v;
      P.rev0 = r;
    }
  }
  // a single trie's views are kernel parameters (not the clique passes'), and
  // the planner clears its control block: no copy
  const bool copied = n > 1 || !tries[0]->rev_entries || query == EH_QUERY_CLIQUE4 || (annot && !hits);
  if (copied) EH_CUDA(cudaMemcpyAsync(base, host, head_bytes, cudaMemcpyHostToDevice, s));
  for (uint32_t g = 0; g < n; g++) {
    const eh_trie* t = tries[g];
    if (!t->rev_entries) continue;
    // every shard of a 4-clique that is split by rows (CliqueShare) runs all the items
    const bool by_rows = hits || P.hits.share.count > 1;
    // records are per entry, only these kernels look rows up, and few entries
    // are better spread over the warps (ER-16K, three entries a warp: 77 us a
    // query against 87 with shared items)
    shape.merge = merge && (hits || blocks_query) && t->n_head < kMerged && head_items > 4 * slots;
    PlanArgs pa{t->view(), rev_view(t), shape, g, by_rows ? 0 : ep.shard_index, by_rows ? 1 : ep.shard_count,
                reinterpret_cast<uint64_t*>(base + o_pos), nullptr};
    pa.tiles = pa.pos + t->n_head;
    if (t->work_pred.p && t->pred_per_probe > 0) {
      pa.ps.pred = t->work_pred.p;
      pa.ps.unit = t->pred_per_probe * shape.chunk;
    }
    const int tiles = ceil_div(t->n_head, kPlanTile);
    unsigned long long* total = &P.ctl->spare[1];
    plan_split_kernel<<<tiles, 256, 0, s>>>(pa, P.ctl, copied ? 0 : (uint32_t)P.ctl_bytes());
    plan_place_kernel<<<tiles, 256, 0, s>>>(pa, total, P.ctl);
    const uint64_t most = std::min<uint64_t>(t->n_head, t->rev_entries) +
                          (t->rev_pairs + kRowCost * t->rev_entries) / ep.chunk;
    plan_fill_kernel<<<(int)std::min<uint64_t>(num_sms() * 8, (most + 255) / 256), 256, 0, s>>>(pa, total, P.ctl,
                                                                                              P.items, P.bitems);
    EH_CHECK_LAUNCH();
    P.plan_launches += 3;
  }
  const uint64_t units = P.cap_b + (P.cap_w + ep.warps - 1) / ep.warps;
  P.grid = (int)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)num_sms() * per_sm, units));
  if (P.entries && annot && !hits && n == 1 && tries[0]->dir == DIR_SYM)
    P.plan_launches += hot_sets(ctx, tries[0], P.hot);
  if (query == EH_QUERY_CLIQUE4 && !hits && ep.s_cap) {
    // one S buffer per resident warp, at most 2 GiB in all
    const uint64_t per_block = (uint64_t)ep.warps * ep.s_cap * 4;
    P.grid = std::max(1, (int)std::min<uint64_t>((uint64_t)P.grid, (2ull << 30) / per_block));
    P.gs.alloc((size_t)P.grid * ep.warps * ep.s_cap, s);
  }
  P.ep = ep;
  P.ep.held = nullptr;
}

// Enqueue one run of a prepared launch; the first follows prepare directly, a
// later one resets the queues.  No host synchronisation: capturable in a CUDA
// graph.  Returns the kernels launched.
static uint32_t launch(eh_context* ctx, Prepared& P, unsigned long long* d_total, unsigned long long* d_annot,
                   float* d_records, bool again = false) {
  cudaStream_t s = ctx->stream;
  if (!P.entries) return 0;
  if (again) EH_CUDA(cudaMemsetAsync(P.ctl->queue, 0, 8, s));
  const ExecParams& ep = P.ep;
  if (P.hits.on) {
    const Hits& H = P.hits;
    const HitsView hv = H.view();
    EH_CUDA(cudaMemsetAsync(H.mask.p, 0, H.words * 4, s));
    (P.n == 1 ? hits_kernel<true> : hits_kernel<false>)<<<P.grid, P.threads, P.smem, s>>>(
        P.view0, P.rev0, P.dv, P.dr, P.items, P.ctl->items, ep.smem_words, P.ctl->queue, hv, d_records);
    EH_CHECK_LAUNCH();
    uint32_t launches = 1;
    if (H.use == HITS_CLIQUE) {
      const uint32_t most = num_sms() * 8, span = std::min(32u, std::max(1u, H.heads / (8 * most)));
      clique_small_kernel<<<std::min<int>(most, ceil_div(H.heads, 8 * span)), 256, 0, s>>>(P.dv, hv, span, d_total);
      EH_CHECK_LAUNCH();
      launches++;
      if (H.units) {
        const uint32_t warps = 8 * most, grab = std::min(4u, std::max(1u, H.units / warps));
        const uint32_t slices = std::min(8u, std::max(1u, warps / H.units));
        const uint64_t turns = (uint64_t)H.units * slices / grab + 1;
        (slices > 1 ? clique_big_kernel<true> : clique_big_kernel<false>)<<<
            (int)std::min<uint64_t>(most, ceil_div(turns, 8)), 256, 0, s>>>(P.dv, hv, H.units, grab, slices,
                                                                           P.ctl->queue + 1, d_total);
        EH_CHECK_LAUNCH();
        launches++;
        if (H.longest > 32 * kSparseWords) {
          EH_CUDA(cudaMemsetAsync(H.heavy.p, 0, 8, s));
          EH_CUDA(cudaMemsetAsync(H.heavy.p + 2, 0xff, (H.heavy.n - 2) * 4, s));
          const HeavyUnits heavy{H.heavy.p, H.heavy.p + 2, (uint32_t)H.heavy.n - 2};
          clique_wide_kernel<<<num_sms() * 4, 256, 0, s>>>(P.dv, hv, H.units, heavy, d_total);
          EH_CHECK_LAUNCH();
          launches++;
        }
      }
    } else if (H.use == HITS_ANNOT && H.units) {
      const bool wide_parts = H.longest > kWidePart;
      const uint32_t blocks = num_sms() * 8, run = std::min(16u, std::max(1u, H.units / (8 * blocks)));
      annot_hits_kernel<false><<<blocks, 256, 0, s>>>(P.view0, hv, H.units, run, d_annot);
      if (wide_parts) annot_hits_kernel<true><<<blocks, 256, 0, s>>>(P.view0, hv, H.units, run, d_annot);
      EH_CHECK_LAUNCH();
      launches += wide_parts ? 2 : 1;
    }
    return launches;
  }
  QueryOut out{ep.long_row, d_total, d_annot, d_records, P.ctl->queue, P.ctl->items, P.bitems};
  out.sel = P.sel;
  for (int k = 0; k < kHot; k++) out.hot[k] = P.hot[k];
  out.gsbuf = ep.s_cap ? P.gs.p : nullptr;
  out.gcap = ep.s_cap;
  out.share = P.hits.share;
  if (P.query == EH_QUERY_CLIQUE4)
    clique4_kernel<<<P.grid, P.threads, P.smem, s>>>(P.dv, P.dr, P.items, ep.smem_words, out);
  else if (P.annot)
    triangle_kernel<MODE_ANNOT, true><<<P.grid, P.threads, P.smem, s>>>(P.view0, P.rev0, P.dv, P.dr, P.items,
                                                                        ep.smem_words, out);
  else if (P.n == 1)
    triangle_kernel<MODE_COUNT, true><<<P.grid, P.threads, P.smem, s>>>(P.view0, P.rev0, P.dv, P.dr, P.items,
                                                                        ep.smem_words, out);
  else
    triangle_kernel<MODE_COUNT, false><<<P.grid, P.threads, P.smem, s>>>(P.view0, P.rev0, P.dv, P.dr, P.items,
                                                                         ep.smem_words, out);
  EH_CHECK_LAUNCH();
  return 1;
}

// Plan and run; nothing is waited for.  ev1 and ev2 bracket the intersection
// kernels.  Results go to P.total (spare: nowhere that is read).  rec: one record per
// item, of the plan that runs otherwise but for items that entries share (a record is
// one set's).
static Launch run_plans(eh_context* ctx, const eh_trie* const* tries, uint32_t n, int query, ExecParams ep,
                        bool annot, Prepared& P, unsigned long long* d_annot, DevBuf<float>* rec = nullptr,
                        const uint32_t* sel = nullptr, bool spare = false) {
  cudaStream_t s = ctx->stream;
  Launch L;
  {
    TracePhase ph("query.prepare", s);
    // selections weight cliques by their members: they run without masks
    const int use = sel ? -1 : query == EH_QUERY_CLIQUE4 ? HITS_CLIQUE : annot ? HITS_ANNOT : -1;
    prepare(ctx, tries, n, query, ep, annot, P, true, use, false, rec == nullptr);
  }
  if (rec) rec->alloc(8 * (P.cap_w + P.cap_b), s);
  P.sel = sel;
  L.launches = P.plan_launches;
  EH_CUDA(cudaEventRecord(ctx->ev1, s));
  {
    TracePhase ph("query.kernel", s);
    L.launches += launch(ctx, P, spare ? P.ctl->spare : P.total, d_annot, rec ? rec->p : nullptr);
  }
  EH_CUDA(cudaEventRecord(ctx->ev2, s));
  return L;
}

// The control block and results of a run, once everything before is done; the
// query's device time.
struct Returned {
  const Control* ctl;
  const unsigned long long* total;
  uint64_t items;
  float query_ms, kernel_ms;
};
static Returned finish(eh_context* ctx, const Prepared& P) {
  cudaStream_t s = ctx->stream;
  unsigned char* host = pinned(ctx, P.ctl_bytes());
  EH_CUDA(cudaMemcpyAsync(host, P.ctl, P.ctl_bytes(), cudaMemcpyDeviceToHost, s));
  EH_CUDA(cudaEventRecord(ctx->ev3, s));
  EH_CUDA(cudaEventSynchronize(ctx->ev3));
  Returned r{reinterpret_cast<const Control*>(host),
             reinterpret_cast<const unsigned long long*>(host + sizeof(Control)), 0, 0, 0};
  r.items = (uint64_t)r.ctl->items[0] + r.ctl->items[1];
  EH_CUDA(cudaEventElapsedTime(&r.query_ms, ctx->ev0, ctx->ev3));
  if (P.entries) EH_CUDA(cudaEventElapsedTime(&r.kernel_ms, ctx->ev1, ctx->ev2));
  return r;
}

// Algorithmic bytes of the triangle plan: both uint32 inputs of every
// pairwise intersection the reference loop nest evaluates, read once each:
// 4 * sum over rows (a,b) of (d(a) + d(b)) = 4 * (sum_a d(a)^2 + wedges).
static uint64_t triangle_algorithmic_bytes(const eh_trie* t) { return 4 * (t->sum_sq_deg + t->total_wedges); }

static void fill_stats(eh_query_stats* st, float query_ms, float kernel_ms, uint32_t launches, uint64_t items,
                       uint64_t pairs, uint64_t alg) {
  if (!st) return;
  st->query_ms = query_ms;
  st->kernel_ms = kernel_ms;
  st->launches = launches;
  st->work_items = items;
  st->wedges = pairs;
  st->algorithmic_bytes = alg;
}

// The root bag of the lollipop / barbell plans over a per-head-entry
// annotation T (the annotated bag's z, by head position of t; Tv: the same
// by node value, or null to derive it): LollipopAgg sum_a T(a) * |N(a)|,
// BarbellAgg sum_a T(a) * sum_{x in N(a)} Tv(x).  Adds into total[0];
// returns the kernels launched.
static uint32_t root_bag(eh_context* ctx, const eh_trie* t, int query, const unsigned long long* T,
                         const unsigned long long* Tv, unsigned long long* total) {
  cudaStream_t s = ctx->stream;
  if (!t->n_head) return 0;
  uint32_t launches = 0;
  if (query == EH_QUERY_LOLLIPOP) {
    root_kernel<false><<<num_sms() * 8, 256, 0, s>>>(t->view(), T, nullptr, total, nullptr, nullptr);
    EH_CHECK_LAUNCH();
    return 1;
  }
  DevBuf<unsigned long long> tv;
  if (!Tv) {
    tv.alloc(t->n_nodes ? t->n_nodes : 1, s);
    t_by_value_kernel<<<num_sms() * 8, 256, 0, s>>>(t->view(), T, tv.p);
    EH_CHECK_LAUNCH();
    Tv = tv.p;
    launches++;
  }
  DevBuf<uint32_t> big;
  const bool has_big = t->info.max_set > kRootBig;
  if (has_big) {
    big.alloc((size_t)t->n_head + 1, s);  // their number, then the entries
    EH_CUDA(cudaMemsetAsync(big.p, 0, 4, s));
  }
  root_kernel<true><<<num_sms() * 8, 256, 0, s>>>(t->view(), T, Tv, total, big.p + 1, big.p);
  EH_CHECK_LAUNCH();
  launches++;
  if (has_big) {
    root_big_kernel<<<num_sms() * 4, 256, 0, s>>>(t->view(), big.p + 1, big.p, T, Tv, total);
    EH_CHECK_LAUNCH();
    launches++;
  }
  return launches;
}

// z by node value (zero beyond n_values) -> the same by head position
__global__ void z_by_head_kernel(TrieView t, const unsigned long long* __restrict__ zv, uint32_t n_values,
                                 unsigned long long* __restrict__ T) {
  for (uint32_t a = blockIdx.x * blockDim.x + threadIdx.x; a < t.n_head; a += gridDim.x * blockDim.x) {
    const uint32_t v = t.head[a];
    T[a] = v < n_values ? zv[v] : 0ull;
  }
}

// The root bag of lollipop / barbell over an annotation z given by value on
// the host (the generated root bags of an annotated intermediate,
// EHGenerator.scala:399-480 with TrieIterator::get_annotation,
// TrieIterator.cpp:45-59): LOLLIPOP sum_a z(a) |N(a)|, BARBELL
// sum_{(a,x)} z(a) z(x), modulo 2^64.
void query_weighted_root(eh_context* ctx, const eh_trie* t, int query, const uint64_t* z, uint32_t n_values,
                         uint64_t* result) {
  cudaStream_t s = ctx->stream;
  EH_REQUIRE(query == EH_QUERY_LOLLIPOP || query == EH_QUERY_BARBELL, EH_ERR_INVALID,
             "the weighted root bag is EH_QUERY_LOLLIPOP or EH_QUERY_BARBELL");
  EH_REQUIRE(t->ctx == ctx, EH_ERR_INVALID, "trie belongs to another context");
  EH_REQUIRE(n_values == 0 || z, EH_ERR_INVALID, "null annotation");
  const uint32_t nv = std::min(n_values, t->n_nodes);
  DevBuf<unsigned long long> zv(nv ? nv : 1, s), T(t->n_head ? t->n_head : 1, s), total(1, s);
  EH_CUDA(cudaMemsetAsync(total.p, 0, 8, s));
  if (nv) EH_CUDA(cudaMemcpyAsync(zv.p, z, 8ull * nv, cudaMemcpyHostToDevice, s));
  if (t->n_head) {
    z_by_head_kernel<<<num_sms() * 4, 256, 0, s>>>(t->view(), zv.p, nv, T.p);
    EH_CHECK_LAUNCH();
    if (query == EH_QUERY_BARBELL) {
      // Tv over the whole value domain: values of the relation outside its head still carry z
      DevBuf<unsigned long long> tv(t->n_nodes ? t->n_nodes : 1, s);
      EH_CUDA(cudaMemsetAsync(tv.p, 0, (size_t)(t->n_nodes ? t->n_nodes : 1) * 8, s));
      if (nv) EH_CUDA(cudaMemcpyAsync(tv.p, zv.p, 8ull * nv, cudaMemcpyDeviceToDevice, s));
      root_bag(ctx, t, query, T.p, tv.p, total.p);
      unsigned long long h = 0;
      EH_CUDA(cudaMemcpyAsync(&h, total.p, 8, cudaMemcpyDeviceToHost, s));
      EH_CUDA(cudaStreamSynchronize(s));
      *result = h;
      return;
    }
    root_bag(ctx, t, query, T.p, nullptr, total.p);
  }
  unsigned long long h = 0;
  EH_CUDA(cudaMemcpyAsync(&h, total.p, 8, cudaMemcpyDeviceToHost, s));
  EH_CUDA(cudaStreamSynchronize(s));
  *result = h;
}

// The annotated pass's per-head counters take one global atomic per hit
// (2.8 G on Chung-Lu 2^23).  Measured on B200 (Chung-Lu 2^23 lollipop): with
// the counters in the stream-ordered pool the pass ran at 243 or 184 ms
// depending on where the pool placed them (holding a 128 MB allocation before
// the query flipped it); in an allocation of their own from cudaMalloc it ran
// at 184 ms whatever the pool held.  The context keeps one such buffer, grown
// (with the stream drained first) when a larger trie needs it.
static unsigned long long* annot_buffer(eh_context* ctx, size_t n) {
  if (n > ctx->annot_cap) {
    EH_CUDA(cudaStreamSynchronize(ctx->stream));
    if (ctx->annot) EH_CUDA(cudaFree(ctx->annot));
    ctx->annot = nullptr;
    ctx->annot_cap = 0;
    if (cudaMalloc((void**)&ctx->annot, n * sizeof(unsigned long long)) != cudaSuccess) {
      cudaGetLastError();
      ctx->annot = nullptr;
      throw Error{EH_ERR_OOM, "device allocation of " + std::to_string(n * 8) + " bytes failed"};
    }
    ctx->annot_cap = n;
  }
  return ctx->annot;
}

static void run_count(eh_context* ctx, const eh_trie* const* tries, uint32_t n, int query, bool record, ExecParams ep,
                      uint64_t* results, eh_query_stats* stats) {
  cudaStream_t s = ctx->stream;
  Prepared P;
  Launch L;
  DevBuf<float> rec;
  DevBuf<float>* recorded = record ? &rec : nullptr;
  if (query == EH_QUERY_TRIANGLE || query == EH_QUERY_CLIQUE4) {
    L = run_plans(ctx, tries, n, query, ep, false, P, nullptr, recorded);
  } else {
    EH_REQUIRE(n == 1, EH_ERR_UNSUPPORTED, "batched lollipop/barbell is not supported");
    const eh_trie* t = tries[0];
    EH_REQUIRE(ep.shard_count == 1, EH_ERR_UNSUPPORTED, "lollipop/barbell run unsharded");
    unsigned long long* T = annot_buffer(ctx, t->n_head ? t->n_head : 1);
    EH_CUDA(cudaMemsetAsync(T, 0, (t->n_head ? t->n_head : 1) * 8, s));
    // the annotated pass (recorded), then the root bag over T into P.total
    L = run_plans(ctx, tries, 1, EH_QUERY_TRIANGLE, ep, true, P, T, recorded, nullptr, true);
    L.launches += root_bag(ctx, t, query, T, nullptr, P.total);
  }
  const Returned got = finish(ctx, P);
  const unsigned long long* h = got.total;
  for (uint32_t g = 0; g < n; g++) {
    uint64_t v = h[g];
    const int dir = tries[g]->dir;
    // on a symmetric relation every undirected triangle is found once (rows
    // a<b) and the reference counts each of its 3! orderings; 4! for 4-cliques
    if (dir == DIR_SYM && query == EH_QUERY_TRIANGLE) v *= 6ull;
    if (dir == DIR_SYM && query == EH_QUERY_CLIQUE4) v *= 24ull;
    results[g] = v;
  }
  if (record) {
    ctx->timing_records.resize(8 * (size_t)got.items);
    if (got.items)
      EH_CUDA(cudaMemcpy(ctx->timing_records.data(), rec.p, 8 * (size_t)got.items * sizeof(float),
                         cudaMemcpyDeviceToHost));
  }
  uint64_t alg = 0;
  for (uint32_t g = 0; g < n; g++) alg += triangle_algorithmic_bytes(tries[g]);
  fill_stats(stats, got.query_ms, got.kernel_ms, L.launches, got.items, P.pairs, alg);
}

void query_count_batched(eh_context* ctx, const eh_trie* const* tries, uint32_t n, int query,
                         const eh_exec_config* cfg, uint64_t* results, eh_query_stats* stats) {
  EH_REQUIRE(query >= EH_QUERY_TRIANGLE && query <= EH_QUERY_BARBELL, EH_ERR_INVALID, "unknown query");
  EH_REQUIRE(n > 0, EH_ERR_INVALID, "no tries");
  for (uint32_t g = 0; g < n; g++) {
    EH_REQUIRE(tries[g] != nullptr, EH_ERR_INVALID, "null trie");
    EH_REQUIRE(tries[g]->ctx == ctx, EH_ERR_INVALID, "trie belongs to another context");
  }
  const ExecParams ep = exec_params(cfg);
  const bool record = cfg && cfg->record_timings && n == 1;
  Call call(ctx);
  TracePhase ph_all("query.total", ctx->stream);
  EH_CUDA(cudaEventRecord(ctx->ev0, ctx->stream));
  with_or_without_masks(ctx, ep, [&](const ExecParams& p) { run_count(ctx, tries, n, query, record, p, results, stats); });
}

void query_count(eh_context* ctx, const eh_trie* t, int query, const eh_exec_config* cfg, uint64_t* result,
                 eh_query_stats* stats) {
  const eh_trie* ts[1] = {t};
  query_count_batched(ctx, ts, 1, query, cfg, result, stats);
}

void triangle_annotation(eh_context* ctx, const eh_trie* t, const eh_exec_config* cfg, uint64_t* annot_dev) {
  cudaStream_t s = ctx->stream;
  ExecParams ep = exec_params(cfg);
  ep.shard_index = 0;
  ep.shard_count = 1;
  Call call(ctx);
  const eh_trie* ts[1] = {t};
  with_or_without_masks(ctx, ep, [&](const ExecParams& p) {
    EH_CUDA(cudaMemsetAsync(annot_dev, 0, (t->n_head ? t->n_head : 1) * 8, s));
    Prepared P;
    run_plans(ctx, ts, 1, EH_QUERY_TRIANGLE, p, true, P, (unsigned long long*)annot_dev, nullptr, nullptr, true);
    EH_CUDA(cudaStreamSynchronize(s));
  });
}

// ------------------------------------------------------------ selections
// An equality selection x = v on an attribute with one accessor is answered
// at the head of its relation (emitHeadContainsSelections,
// EHGenerator.scala:681-701): the selected bag holds the partners of v with
// annotation 1 each.  Edge(a,x) in order [x,a] gives
// partners(v) = {a : (a,v) ∈ Edge}: the head entries whose child set holds
// v.  One thread per head entry binary-searches v in its sorted list (kept
// whatever the set's layout).
//   bits: optional bitmap over node values, set for every partner a;
//   T:    optional per-head annotation, summed over the partners into
//         sums[0] and over N(v) ∩ head into sums[1];
//   sums[2] counts the partners.
__global__ void select_partners_kernel(TrieView t, uint32_t v, uint32_t* __restrict__ bits,
                                       const unsigned long long* __restrict__ T,
                                       unsigned long long* __restrict__ sums) {
  const uint32_t stride = gridDim.x * blockDim.x;
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long s_in = 0, s_out = 0, n_in = 0;
  for (uint32_t i = tid; i < t.n_head; i += stride) {
    const uint64_t end = t.off[i + 1];
    uint64_t lo = t.off[i], hi = end;
    while (lo < hi) {
      const uint64_t mid = (lo + hi) >> 1;
      if (__ldg(t.vals + mid) < v) lo = mid + 1; else hi = mid;
    }
    if (lo < end && __ldg(t.vals + lo) == v) {
      n_in++;
      if (bits) {
        const uint32_t a = t.head[i];
        atomicOr(bits + (a >> 5), 1u << (a & 31));
      }
      if (T) s_in += T[i];
    }
  }
  if (T && v < t.n_nodes) {
    const int32_t hv = t.head_index[v];
    if (hv >= 0)
      for (uint64_t e = t.off[hv] + tid; e < t.off[hv + 1]; e += stride) {
        const int32_t hx = __ldg(t.head_index + __ldg(t.vals + e));
        if (hx >= 0) s_out += T[hx];
      }
  }
  s_in = warp_sum(s_in);
  s_out = warp_sum(s_out);
  n_in = warp_sum(n_in);
  if (lane_id() == 0) {
    if (s_in) atomicAdd(sums, s_in);
    if (s_out) atomicAdd(sums + 1, s_out);
    if (n_in) atomicAdd(sums + 2, n_in);
  }
}

// FliqueSelAgg(;z) :- 4-clique(a,b,c,d), Edge(a,x), x=v and
// BarbellSelAgg(;w) :- triangle(a,b,c), Edge(a,p), Edge(p,x),
// triangle(x,y,z), p=v (test/graph/travis.py:385-401, 472-487; plans
// QueryPlannerTest.scala:230-304).
//  4-clique: the 4-clique plan with its roots restricted to partners(v).
//  Barbell: bag_1_x_y_z reduces to the scalar sum_{x ∈ N(v)} T(x) and the
//  root bag to sum_{a ∈ partners(v)} T(a) times it, T the triangle
//  annotation of the lollipop/barbell bag.
void query_count_select(eh_context* ctx, const eh_trie* t, int query, uint32_t value, const eh_exec_config* cfg,
                        uint64_t* result, eh_query_stats* stats) {
  cudaStream_t s = ctx->stream;
  EH_REQUIRE(query == EH_QUERY_CLIQUE4_SEL || query == EH_QUERY_BARBELL_SEL, EH_ERR_INVALID,
             "selection queries are EH_QUERY_CLIQUE4_SEL and EH_QUERY_BARBELL_SEL");
  EH_REQUIRE(t->ctx == ctx, EH_ERR_INVALID, "trie belongs to another context");
  ExecParams ep = exec_params(cfg);
  EH_REQUIRE(ep.shard_count == 1, EH_ERR_UNSUPPORTED, "selection plans run unsharded");
  const bool clique = query == EH_QUERY_CLIQUE4_SEL;
  Call call(ctx);
  EH_CUDA(cudaEventRecord(ctx->ev0, s));
  DevBuf<unsigned long long> sums(4, s);  // partner sum, N(v) sum, partners, plan total
  EH_CUDA(cudaMemsetAsync(sums.p, 0, 32, s));
  const uint64_t nbits = t->n_nodes ? ((uint64_t)t->n_nodes + 31) / 32 : 1;
  DevBuf<uint32_t> bits;
  if (clique) {
    bits.alloc(nbits, s);
    EH_CUDA(cudaMemsetAsync(bits.p, 0, nbits * 4, s));
  }
  const int sgrid = num_sms() * 8;
  Launch L;
  if (t->n_head) {
    select_partners_kernel<<<sgrid, 256, 0, s>>>(t->view(), value, clique ? bits.p : nullptr, nullptr, sums.p);
    EH_CHECK_LAUNCH();
    L.launches++;
  }
  // Encoding::value_to_key.at(v) throws for a value in neither column
  int32_t hv = -1;
  if (value < t->n_nodes)
    EH_CUDA(cudaMemcpyAsync(&hv, t->head_index.p + value, 4, cudaMemcpyDeviceToHost, s));
  unsigned long long h[4] = {0, 0, 0, 0};
  EH_CUDA(cudaMemcpyAsync(h, sums.p, 32, cudaMemcpyDeviceToHost, s));
  EH_CUDA(cudaStreamSynchronize(s));
  EH_REQUIRE(hv >= 0 || h[2] > 0, EH_ERR_INVALID,
             "selection value " + std::to_string(value) + " is not in the relation");
  uint64_t items = 0, pairs = 0;
  float kernel_ms = 0;
  const eh_trie* ts[1] = {t};
  uint64_t v = 0;
  if (h[2] > 0) {  // no partners: the selected bag is empty and so is the join
    if (clique) {
      Prepared P;
      L.launches += run_plans(ctx, ts, 1, EH_QUERY_CLIQUE4, ep, false, P, nullptr, nullptr, bits.p).launches;
      const Returned got = finish(ctx, P);
      items = got.items;
      pairs = P.pairs;
      kernel_ms = got.kernel_ms;
      v = got.total[0];
      if (t->dir == DIR_SYM) v *= 6ull;  // 3! orderings start at each selected member
    } else if (hv >= 0) {
      DevBuf<unsigned long long> T(t->n_head, s);
      with_or_without_masks(ctx, ep, [&](const ExecParams& p) {
        EH_CUDA(cudaMemsetAsync(T.p, 0, (size_t)t->n_head * 8, s));
        EH_CUDA(cudaMemsetAsync(sums.p, 0, 32, s));
        Prepared P;
        const Launch K = run_plans(ctx, ts, 1, EH_QUERY_TRIANGLE, p, true, P, T.p, nullptr, nullptr, true);
        select_partners_kernel<<<sgrid, 256, 0, s>>>(t->view(), value, nullptr, T.p, sums.p);
        EH_CHECK_LAUNCH();
        L.launches += K.launches + 1;
        EH_CUDA(cudaMemcpyAsync(h, sums.p, 32, cudaMemcpyDeviceToHost, s));
        const Returned got = finish(ctx, P);
        items = got.items;
        pairs = P.pairs;
        kernel_ms = got.kernel_ms;
      });
      v = (uint64_t)h[0] * (uint64_t)h[1];
    }
  }
  EH_CUDA(cudaEventRecord(ctx->ev2, s));
  EH_CUDA(cudaEventSynchronize(ctx->ev2));
  float qms = 0;
  EH_CUDA(cudaEventElapsedTime(&qms, ctx->ev0, ctx->ev2));
  *result = v;
  fill_stats(stats, qms, kernel_ms, L.launches, items, pairs, triangle_algorithmic_bytes(t));
}

// ------------------------------------------------------------ materialize
// Triangle(a,b,c) :- Edge(a,b),Edge(b,c),Edge(a,c) as tuples sorted by
// (a,b,c): the rows Trie::foreach (Trie.cpp:130-160) yields on the
// reference's materialized output trie (TrieBuilder::build_set /
// allocate_next / set_level, TrieBuilder.cpp:44-221, 376-410).  An up or down
// relation's come in order from its hit masks (materialize_hits).  Of a symmetric or
// general one, and where there is no memory for masks, one counting run sizes every
// work item's slice, a second run writes the tuples into the slices, and two stable
// key-value radix sorts (by c, then by (a,b)) order them.
__global__ void iota_kernel(uint32_t* __restrict__ v, uint64_t n) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    v[i] = (uint32_t)i;
}
__global__ void widen_kernel(const uint32_t* __restrict__ c, uint64_t n, uint64_t* __restrict__ k) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    k[i] = c[i];
}
// keys2[i] = a[idx[i]] << bb | b[idx[i]], vals2[i] = c value (keys1[i])
__global__ void ab_key_kernel(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b,
                              const uint32_t* __restrict__ idx, const uint64_t* __restrict__ csorted, uint64_t n,
                              int bb, uint64_t* __restrict__ keys, uint32_t* __restrict__ vals) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t j = idx[i];
    keys[i] = ((uint64_t)a[j] << bb) | b[j];
    vals[i] = (uint32_t)csorted[i];
  }
}
// triangle i at out[i * stride], its next value `next` further
__global__ void split_abc_kernel(const uint64_t* __restrict__ keys, const uint32_t* __restrict__ c, uint64_t n, int bb,
                                 int stride, uint64_t next, uint32_t* __restrict__ out) {
  const uint64_t mask = (1ull << bb) - 1;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t* o = out + i * stride;
    o[0] = (uint32_t)(keys[i] >> bb);
    o[next] = (uint32_t)(keys[i] & mask);
    o[2 * next] = c[i];
  }
}

// TriangleProj(a,b): the reference's plan drops attributes that are neither
// materialized, selected nor aggregated (codegen/query/QueryPlan.scala:245),
// so c is never intersected: the rows are (a,b) with b in N(a) ∩ head, in
// trie order.  One flag + scan + compact over the rows.
__global__ void proj_flag_kernel(TrieView t, uint32_t* __restrict__ flag) {
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < t.rows; e += (uint64_t)gridDim.x * blockDim.x)
    flag[e] = __ldg(t.head_index + t.vals[e]) >= 0 ? 1u : 0u;
}
__global__ void proj_write_kernel(TrieView t, const uint32_t* __restrict__ seg, const uint32_t* __restrict__ pos,
                                  uint32_t* __restrict__ a, uint32_t* __restrict__ b) {
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < t.rows; e += (uint64_t)gridDim.x * blockDim.x)
    if (__ldg(t.head_index + t.vals[e]) >= 0) {
      a[pos[e]] = t.head[seg[e]];
      b[pos[e]] = t.vals[e];
    }
}
__global__ void seg_of_rows_kernel(const uint64_t* __restrict__ off, uint32_t nh, uint32_t* __restrict__ seg) {
  const uint32_t lane = lane_id();
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t i = warp; i < nh; i += nwarps)
    for (uint64_t e = off[i] + lane; e < off[i + 1]; e += 32) seg[e] = i;
}

static void query_project_ab(eh_context* ctx, const eh_trie* t, uint32_t* ha, uint32_t* hb, uint64_t cap,
                             uint64_t* n_rows) {
  cudaStream_t s = ctx->stream;
  *n_rows = 0;
  if (!t->rows) return;
  const int grid = num_sms() * 8;
  DevBuf<uint32_t> pos(t->rows, s), seg(t->rows, s), tot(1, s);
  proj_flag_kernel<<<grid, 256, 0, s>>>(t->view(), pos.p);
  EH_CHECK_LAUNCH();
  exclusive_scan<uint32_t>(pos.p, pos.p, t->rows, tot.p, s);
  uint32_t m = 0;
  EH_CUDA(cudaMemcpyAsync(&m, tot.p, 4, cudaMemcpyDeviceToHost, s));
  EH_CUDA(cudaStreamSynchronize(s));
  *n_rows = m;
  if (!ha || !hb || !m) return;
  EH_REQUIRE(cap >= m, EH_ERR_INVALID, "output columns hold fewer rows than the result");
  DevBuf<uint32_t> da(m, s), db(m, s);
  seg_of_rows_kernel<<<grid, 256, 0, s>>>(t->off.p, t->n_head, seg.p);
  proj_write_kernel<<<grid, 256, 0, s>>>(t->view(), seg.p, pos.p, da.p, db.p);
  EH_CHECK_LAUNCH();
  EH_CUDA(cudaMemcpyAsync(ha, da.p, (size_t)m * 4, cudaMemcpyDeviceToHost, s));
  EH_CUDA(cudaMemcpyAsync(hb, db.p, (size_t)m * 4, cudaMemcpyDeviceToHost, s));
  EH_CUDA(cudaStreamSynchronize(s));
}

// Where materialized triangles go on the host: three columns, or rows of three.
struct HostRows {
  uint32_t *a, *b, *c;
  uint32_t* rows;  // null: the columns
  bool given() const { return rows || (a && b && c); }
  void take(const uint32_t* dev, uint64_t n, cudaStream_t s) const {  // n triangles, laid out the same way
    if (rows) {
      EH_CUDA(cudaMemcpyAsync(rows, dev, 3 * n * 4, cudaMemcpyDeviceToHost, s));
    } else {
      EH_CUDA(cudaMemcpyAsync(a, dev, n * 4, cudaMemcpyDeviceToHost, s));
      EH_CUDA(cudaMemcpyAsync(b, dev + n, n * 4, cudaMemcpyDeviceToHost, s));
      EH_CUDA(cudaMemcpyAsync(c, dev + 2 * n, n * 4, cudaMemcpyDeviceToHost, s));
    }
    EH_CUDA(cudaStreamSynchronize(s));
  }
};

// Oriented relations: the hit masks hold every triangle at its place in the
// order (a, b, c), so the rows are counted per relation row, placed by a scan
// and written in order; nothing is sorted.  false: no masks for this relation.
static bool materialize_hits(eh_context* ctx, const eh_trie* t, const ExecParams& ep, const HostRows& host,
                             uint64_t cap, uint64_t* n_rows) {
  cudaStream_t s = ctx->stream;
  Prepared P;
  const eh_trie* ts[1] = {t};
  prepare(ctx, ts, 1, EH_QUERY_TRIANGLE, ep, false, P, false, HITS_ROWS);
  if (!P.hits.on) return false;
  *n_rows = 0;
  if (!P.entries) return true;
  launch(ctx, P, nullptr, nullptr, nullptr);
  DevBuf<uint32_t> seg(t->rows, s);
  DevBuf<uint64_t> pos(t->rows, s), tot(1, s);
  const int grid = num_sms() * 8;
  seg_of_rows_kernel<<<grid, 256, 0, s>>>(t->off.p, t->n_head, seg.p);
  hits_row_count_kernel<<<grid, 256, 0, s>>>(t->view(), t->dir, P.hits.view(), seg.p, pos.p);
  EH_CHECK_LAUNCH();
  exclusive_scan<uint64_t>(pos.p, pos.p, t->rows, tot.p, s);
  uint64_t n = 0;
  EH_CUDA(cudaMemcpyAsync(&n, tot.p, 8, cudaMemcpyDeviceToHost, s));
  EH_CUDA(cudaStreamSynchronize(s));
  *n_rows = n;
  if (!n) return true;
  EH_REQUIRE(cap >= n, EH_ERR_INVALID, "output columns hold fewer rows than the result");
  EH_REQUIRE(n < (1ull << 32), EH_ERR_UNSUPPORTED, "materialized results hold fewer than 2^32 rows");
  DevBuf<uint32_t> out(3 * n, s);
  const uint64_t next = host.rows ? 1 : n;  // from a row's one value to its next
  hits_row_write_kernel<<<grid, 256, 0, s>>>(t->view(), t->dir, P.hits.view(), seg.p, pos.p, n, host.rows ? 3 : 1,
                                             out.p, out.p + next, out.p + 2 * next);
  EH_CHECK_LAUNCH();
  host.take(out.p, n, s);
  return true;
}

void query_materialize(eh_context* ctx, const eh_trie* t, int query, const eh_exec_config* cfg, int n_cols,
                       uint32_t* ha, uint32_t* hb, uint32_t* hc, uint64_t cap, uint64_t* n_rows, uint32_t* rows_out) {
  cudaStream_t s = ctx->stream;
  EH_REQUIRE(query == EH_QUERY_TRIANGLE, EH_ERR_UNSUPPORTED, "materialized output is built for the triangle plan");
  EH_REQUIRE(n_cols == 2 || n_cols == 3, EH_ERR_INVALID, "n_cols must be 3 (a,b,c) or 2 (projection on a,b)");
  EH_REQUIRE(t->ctx == ctx, EH_ERR_INVALID, "trie belongs to another context");
  Call call(ctx);
  if (n_cols == 2) {
    query_project_ab(ctx, t, ha, hb, cap, n_rows);
    return;
  }
  const HostRows host{ha, hb, hc, rows_out};
  if (host.given() && t->dir != DIR_SYM) {
    ExecParams ep = exec_params(cfg);
    ep.shard_index = 0;
    ep.shard_count = 1;
    bool done = false;
    with_or_without_masks(ctx, ep, [&](const ExecParams& p) {
      done = p.masks && materialize_hits(ctx, t, p, host, cap, n_rows);
    });
    if (done) return;
  }
  uint64_t n = 0;
  query_count(ctx, t, EH_QUERY_TRIANGLE, cfg, &n, nullptr);
  *n_rows = n;
  if (n == 0 || !host.given()) return;  // the row count is the triangle count
  EH_REQUIRE(cap >= n, EH_ERR_INVALID, "output columns hold fewer rows than the result");
  EH_REQUIRE(n < (1ull << 32), EH_ERR_UNSUPPORTED, "materialized results hold fewer than 2^32 rows");
  ExecParams ep = exec_params(cfg);
  ep.shard_index = 0;
  ep.shard_count = 1;
  Prepared P;
  const eh_trie* ts[1] = {t};
  prepare(ctx, ts, 1, EH_QUERY_TRIANGLE, ep, false, P, false, -1, false, false);
  dynamic_smem_room((const void*)triangle_kernel<MODE_MAT, true>);
  unsigned int n_items = 0;
  EH_CUDA(cudaMemcpyAsync(&n_items, P.ctl->items, 4, cudaMemcpyDeviceToHost, s));
  EH_CUDA(cudaStreamSynchronize(s));
  DevBuf<unsigned long long> counts(n_items ? n_items : 1, s), offs(n_items ? n_items : 1, s), rows(1, s);
  const uint32_t mult = t->dir == DIR_SYM ? 6u : 1u;
  QueryOut out{P.ep.long_row, P.total, nullptr, nullptr, P.ctl->queue, P.ctl->items, P.bitems};
  out.item_counts = counts.p;
  out.count_mult = mult;
  triangle_kernel<MODE_COUNT, true><<<P.grid, P.threads, P.smem, s>>>(P.view0, P.rev0, P.dv, P.dr, P.items,
                                                                      P.ep.smem_words, out);
  EH_CHECK_LAUNCH();
  exclusive_scan<uint64_t>((const uint64_t*)counts.p, (uint64_t*)offs.p, n_items, (uint64_t*)rows.p, s);
  uint64_t nr = 0;
  EH_CUDA(cudaMemcpyAsync(&nr, rows.p, 8, cudaMemcpyDeviceToHost, s));
  EH_CUDA(cudaStreamSynchronize(s));
  EH_REQUIRE(nr == n, EH_ERR_CUDA, "materialize: counting runs disagree");
  DevBuf<uint32_t> ma(n, s), mb(n, s), mc(n, s);
  out.item_counts = nullptr;
  out.item_off = offs.p;
  out.ma = ma.p;
  out.mb = mb.p;
  out.mc = mc.p;
  EH_CUDA(cudaMemsetAsync(P.ctl->queue, 0, 8, s));
  triangle_kernel<MODE_MAT, true><<<P.grid, P.threads, P.smem, s>>>(P.view0, P.rev0, P.dv, P.dr, P.items,
                                                                    P.ep.smem_words, out);
  EH_CHECK_LAUNCH();
  // order by (a, b, c): stable sort by c, then stable sort by (a, b)
  const int grid = num_sms() * 8;
  const int bb = bits_for(t->n_nodes ? t->n_nodes - 1 : 0);
  DevBuf<uint64_t> k1(n, s), k1t(n, s);
  DevBuf<uint32_t> idx(n, s), idxt(n, s);
  widen_kernel<<<grid, 256, 0, s>>>(mc.p, n, k1.p);
  iota_kernel<<<grid, 256, 0, s>>>(idx.p, n);
  EH_CHECK_LAUNCH();
  radix_sort_kv(k1.p, k1t.p, idx.p, idxt.p, n, bb, s);
  DevBuf<uint64_t> k2(n, s);
  DevBuf<uint32_t> v2(n, s);
  ab_key_kernel<<<grid, 256, 0, s>>>(ma.p, mb.p, idx.p, k1.p, n, bb, k2.p, v2.p);
  EH_CHECK_LAUNCH();
  radix_sort_kv(k2.p, k1t.p, v2.p, idxt.p, n, 2 * bb, s);
  DevBuf<uint32_t> sorted(3 * n, s);
  split_abc_kernel<<<grid, 256, 0, s>>>(k2.p, v2.p, n, bb, rows_out ? 3 : 1, rows_out ? 1 : n, sorted.p);
  EH_CHECK_LAUNCH();
  host.take(sorted.p, n, s);
}

// One triangle / 4-clique COUNT of one trie with every piece of device
// scratch (queue, total, views, planner arrays, scan tile sums, work items,
// and the 4-clique's per-warp S buffers when a set is too large for shared
// memory) carved out of `scratch` (256-byte aligned, `bytes` long):
// allocates nothing.  Throws EH_ERR_UNSUPPORTED when the trie needs more
// scratch.  Every check that can fail before the last one is made before
// the first launch; the last (the work plan's size) after a synchronisation,
// so a failing call leaves no work of its own in flight.
static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

void query_count_in_scratch(eh_context* ctx, const eh_trie* t, int query, const eh_exec_config* cfg,
                            unsigned char* scratch, size_t bytes, uint64_t* result) {
  cudaStream_t s = ctx->stream;
  EH_REQUIRE(query == EH_QUERY_TRIANGLE || query == EH_QUERY_CLIQUE4, EH_ERR_UNSUPPORTED,
             "the allocation-free path runs the triangle and 4-clique plans");
  EH_REQUIRE(t->ctx == ctx, EH_ERR_INVALID, "trie belongs to another context");
  ExecParams ep = exec_params(cfg);
  EH_REQUIRE(ep.shard_count == 1, EH_ERR_UNSUPPORTED, "the allocation-free path runs unsharded");
  const bool clique = query == EH_QUERY_CLIQUE4;
  if (clique) {
    size_clique_staging(ep, t->info.max_set);
  }
  // launch shape and shared memory, checked before anything is launched
  const int threads = 32 * ep.warps;
  const size_t smem = (size_t)ep.smem_words * 4 * ep.warps;
  const void* kfn = clique ? (const void*)clique4_kernel : (const void*)triangle_kernel<MODE_COUNT, true>;
  {
    const size_t room = dynamic_smem_room(kfn);
    EH_REQUIRE(smem <= room, EH_ERR_UNSUPPORTED,
               "shared staging of " + std::to_string(smem) + " bytes per block is above the " + std::to_string(room) +
                   " a block may use");
  }
  const int per_sm = blocks_per_sm(kfn, threads, smem);
  // carve the scratch
  const uint32_t nh = t->n_head;
  const uint64_t scan_elems = scan_scratch_elems(nh);
  const size_t off_ctrl = 0;  // u32 queue[2], u64 total, u32 items[2]
  const size_t off_tv = 256;
  const size_t off_rv = align256(off_tv + sizeof(TrieView));
  const size_t off_nitems = align256(off_rv + sizeof(RevView));
  const size_t off_ipos = align256(off_nitems + 4ull * nh);
  const size_t off_scan = align256(off_ipos + 4ull * nh);
  const size_t off_items = align256(off_scan + 4ull * scan_elems);
  EH_REQUIRE(off_items <= bytes, EH_ERR_UNSUPPORTED,
             "trie too large for the allocation-free path: its planner needs " + std::to_string(off_items) +
                 " bytes of scratch before the work items, the path holds " + std::to_string(bytes));
  unsigned int* queue = reinterpret_cast<unsigned int*>(scratch + off_ctrl);
  unsigned long long* total = reinterpret_cast<unsigned long long*>(scratch + off_ctrl + 8);
  TrieView* dv = reinterpret_cast<TrieView*>(scratch + off_tv);
  RevView* dr = reinterpret_cast<RevView*>(scratch + off_rv);
  uint32_t* nitems = reinterpret_cast<uint32_t*>(scratch + off_nitems);
  uint32_t* ipos = reinterpret_cast<uint32_t*>(scratch + off_ipos);
  uint32_t* tot = reinterpret_cast<uint32_t*>(scratch + off_ctrl + 16);  // items: warp items, no block items
  uint32_t* scan_tmp = reinterpret_cast<uint32_t*>(scratch + off_scan);
  Item* items = reinterpret_cast<Item*>(scratch + off_items);
  // the array keeps the previous call's contents: zero what must start at 0
  EH_CUDA(cudaMemsetAsync(scratch + off_ctrl, 0, 24, s));
  const TrieView hv = t->view();
  const RevView hr = rev_view(t);
  EH_CUDA(cudaMemcpyAsync(dv, &hv, sizeof(TrieView), cudaMemcpyHostToDevice, s));
  EH_CUDA(cudaMemcpyAsync(dr, &hr, sizeof(RevView), cudaMemcpyHostToDevice, s));
  uint32_t n_items = 0;
  const int pgrid = num_sms() * 4;
  if (t->rev_entries) {
    plan_count_kernel<<<pgrid, 256, 0, s>>>(hr, nh, ep.chunk, nitems);
    EH_CHECK_LAUNCH();
    exclusive_scan_scratch<uint32_t>(nitems, ipos, nh, tot, scan_tmp, scan_elems, s);
    EH_CUDA(cudaMemcpyAsync(&n_items, tot, 4, cudaMemcpyDeviceToHost, s));
  }
  EH_CUDA(cudaStreamSynchronize(s));  // nothing of this call is in flight past here
  const size_t items_end = align256(off_items + sizeof(Item) * (size_t)n_items);
  EH_REQUIRE(items_end <= bytes, EH_ERR_UNSUPPORTED,
             "trie too large for the allocation-free path: it needs " + std::to_string(items_end) +
                 " bytes of scratch, the path holds " + std::to_string(bytes));
  int grid = std::max(1, std::min(num_sms() * per_sm, (int)((n_items + ep.warps - 1) / ep.warps)));
  uint32_t* gsbuf = nullptr;
  if (clique && ep.s_cap) {
    // one S buffer of s_cap words per resident warp, after the work items;
    // fewer blocks when the rest of the array holds fewer buffers
    const uint64_t per_block = (uint64_t)ep.warps * ep.s_cap * 4;
    const uint64_t fit = (bytes - items_end) / per_block;
    EH_REQUIRE(fit >= 1, EH_ERR_UNSUPPORTED,
               "4-clique: the largest set (" + std::to_string(t->info.max_set) +
                   " elements) needs S buffers of " + std::to_string(per_block) +
                   " bytes per block, more than the allocation-free path has left");
    grid = (int)std::min<uint64_t>((uint64_t)grid, fit);
    gsbuf = reinterpret_cast<uint32_t*>(scratch + items_end);
  }
  if (n_items) {
    plan_fill_scratch_kernel<<<pgrid, 256, 0, s>>>(hr, nh, nitems, ipos, n_items, 0, items);
    EH_CHECK_LAUNCH();
    QueryOut out{ep.long_row, total, nullptr, nullptr, queue, tot};
    out.gsbuf = gsbuf;
    out.gcap = ep.s_cap;
    if (clique)
      clique4_kernel<<<grid, threads, smem, s>>>(dv, dr, items, ep.smem_words, out);
    else
      triangle_kernel<MODE_COUNT, true><<<grid, threads, smem, s>>>(hv, hr, dv, dr, items, ep.smem_words, out);
    EH_CHECK_LAUNCH();
  }
  unsigned long long h = 0;
  EH_CUDA(cudaMemcpyAsync(&h, total, 8, cudaMemcpyDeviceToHost, s));
  EH_CUDA(cudaStreamSynchronize(s));
  uint64_t v = h;
  if (t->dir == DIR_SYM) v *= clique ? 24ull : 6ull;
  *result = v;
}

}  // namespace eh

// ------------------------------------------------------------------ batches
// A prepared batch: one queue over every trie's work items and the whole
// step captured once as a CUDA graph (zero results, zero queue, persistent
// kernel, results to pinned host memory).  A run is one graph launch.
struct eh_batch {
  eh_context* ctx = nullptr;
  eh::Prepared P;
  unsigned long long* host = nullptr;  // pinned
  std::vector<int> dirs;
  uint32_t n = 0;
  uint64_t items = 0;
  uint32_t launches = 0;  // kernels of a run
  int query = 0;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  ~eh_batch() {
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    if (host) cudaFreeHost(host);
  }
};

namespace eh {

static eh_batch* make_batch(eh_context* ctx, const eh_trie* const* tries, uint32_t n, int query,
                            const ExecParams& ep) {
  cudaStream_t s = ctx->stream;
  auto* b = new eh_batch();
  try {
    b->ctx = ctx;
    b->n = n;
    b->query = query;
    for (uint32_t g = 0; g < n; g++) b->dirs.push_back(tries[g]->dir);
    prepare(ctx, tries, n, query, ep, false, b->P, true, query == EH_QUERY_CLIQUE4 ? HITS_CLIQUE : -1, true);
    unsigned int items[2] = {0, 0};
    EH_CUDA(cudaMemcpyAsync(items, b->P.ctl->items, 8, cudaMemcpyDeviceToHost, s));
    EH_CUDA(cudaMallocHost((void**)&b->host, n * sizeof(unsigned long long)));
    EH_CUDA(cudaStreamSynchronize(s));
    b->items = (uint64_t)items[0] + items[1];
    EH_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    cudaError_t cap = cudaSuccess;
    try {
      EH_CUDA(cudaMemsetAsync(b->P.total, 0, n * 8, s));
      b->launches = launch(ctx, b->P, b->P.total, nullptr, nullptr, true);
      EH_CUDA(cudaMemcpyAsync(b->host, b->P.total, n * 8, cudaMemcpyDeviceToHost, s));
    } catch (...) {
      cudaGraph_t g = nullptr;
      cudaStreamEndCapture(s, &g);
      if (g) cudaGraphDestroy(g);
      throw;
    }
    cap = cudaStreamEndCapture(s, &b->graph);
    EH_CUDA(cap);
    EH_CUDA(cudaGraphInstantiate(&b->exec, b->graph, 0));
  } catch (...) {
    delete b;
    throw;
  }
  return b;
}

eh_batch* batch_create(eh_context* ctx, const eh_trie* const* tries, uint32_t n, int query,
                       const eh_exec_config* cfg) {
  EH_REQUIRE(n > 0, EH_ERR_INVALID, "no tries");
  EH_REQUIRE(query == EH_QUERY_TRIANGLE || query == EH_QUERY_CLIQUE4, EH_ERR_UNSUPPORTED,
             "batches run the triangle or 4-clique plan");
  const ExecParams ep = exec_params(cfg);
  for (uint32_t g = 0; g < n; g++)
    EH_REQUIRE(tries[g] && tries[g]->ctx == ctx, EH_ERR_INVALID, "null trie or trie of another context");
  Call call(ctx);
  eh_batch* b = nullptr;
  with_or_without_masks(ctx, ep, [&](const ExecParams& p) { b = make_batch(ctx, tries, n, query, p); });
  return b;
}

void batch_run(eh_context* ctx, eh_batch* b, uint64_t* results, eh_query_stats* stats) {
  cudaStream_t s = ctx->stream;
  EH_REQUIRE(b->ctx == ctx, EH_ERR_INVALID, "batch belongs to another context");
  Call call(ctx);
  EH_CUDA(cudaEventRecord(ctx->ev0, s));
  EH_CUDA(cudaGraphLaunch(b->exec, s));
  EH_CUDA(cudaEventRecord(ctx->ev2, s));
  EH_CUDA(cudaEventSynchronize(ctx->ev2));
  float ms = 0;
  EH_CUDA(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev2));
  for (uint32_t g = 0; g < b->n; g++) {
    uint64_t v = b->host[g];
    if (b->dirs[g] == DIR_SYM) v *= b->query == EH_QUERY_CLIQUE4 ? 24ull : 6ull;
    results[g] = v;
  }
  if (stats) {
    stats->query_ms = ms;
    stats->kernel_ms = ms;
    stats->launches = b->launches;
    stats->work_items = b->items;
    stats->wedges = b->P.pairs;
    stats->algorithmic_bytes = 0;
  }
}

void batch_free(eh_batch* b) {
  cudaSetDevice(b->ctx->device);
  cudaStream_t s = b->ctx->stream;
  cudaStreamSynchronize(s);
  delete b;
  cudaStreamSynchronize(s);
}

}  // namespace eh
