// Row hit masks: which candidates of every row matched, as bits.
//
// For a row a->b the triangle plan intersects N(b) with the candidates of
// N(a) beyond b.  hits_kernel runs exactly those intersections, on the same
// work items and staged sets as triangle_kernel, and keeps every result as a
// bit at the candidate's position in N(a) instead of only counting it.  The
// rows of one a are then the adjacency matrix of its neighbourhood, and the
// plans that read more than the count work on that matrix alone:
//   4-clique     sum over set bits (i, j) of popc(row_i & row_j)
//   annotation   (symmetric relation) row sums and column sums
//   rows         the set bits in order are the sorted triangles of a
//
// Positions.  part(a) is what the plans read of N(a) (staged_range), d its
// length.  On a relation that goes up, position i is element i of the part; on
// one that goes down, element d - 1 - i; so a row at position i always has the
// candidates i + 1 .. d - 1.  (A general relation has no such order: its
// candidates are the whole N(a), and the plans run without masks.)
// Layout.  W = ceil(d / 32) words per row.  Rows come in blocks of 32; block q
// holds the words q .. W - 1 of its rows, word-major: word k of the 32 rows is
// one 128-byte line, so a warp whose lanes hold 32 rows reads one line per
// word.  The last block stores its d - 32 (W - 1) rows, rounded up to a multiple
// of 8: eight rows' words are always two 16-byte loads.
#pragma once

#include "eh_internal.cuh"

namespace eh {

struct HitsView {
  uint32_t* mask;         // words of every head entry of every graph, zero where nothing matched
  const uint32_t* moff;   // [heads] first word of a head entry
  const uint32_t* upre;   // [heads + 1] first work unit of a head entry (second pass); null: none
  const uint32_t* gstart; // [graphs + 1] first head entry of a graph
  uint32_t n_graphs;
  uint32_t heads;         // of all graphs
  CliqueShare share;      // 4-clique: the rows of this rank
};

__host__ __device__ __forceinline__ uint64_t hits_words(uint64_t d) {
  if (d < 2) return 0;
  const uint64_t W = (d + 31) / 32;
  return 32 * (W * (W + 1) / 2 - 1) + ((d - 32 * (W - 1) + 7) & ~7ull);
}
// steps of the 4-clique's second pass over a full matrix, up to a factor
__host__ __device__ __forceinline__ uint64_t hits_work(uint64_t d) {
  const uint64_t W = (d + 31) / 32;
  return W * W * W;
}
// words before row block q; rows of a block (the stride between two words of a row)
__device__ __forceinline__ uint32_t hits_block(uint32_t q, uint32_t W) { return 32 * (q * W - q * (q - 1) / 2); }
__device__ __forceinline__ uint32_t hits_stride(uint32_t q, uint32_t W, uint32_t d) {
  return q + 1 < W ? 32u : (d - 32u * q + 7) & ~7u;
}

// One batch of 32 rows at a time, a row per lane.  Rows of at least kTripRow
// candidates run as trips: a trip is one mask word of one row, a bit per lane,
// and the trips of all the batch's rows form one list, taken kHitTrips at a
// time (so a row need not fill them) with their candidates loaded before any is
// probed.  Lane t keeps the word of trip t and writes it after 32
// trips.  Shorter rows are flattened over the lanes, and each lane cuts its
// row's bits out of the trip's ballot (a short row's candidates lie in at most
// two words).  Only non-zero words are written.
constexpr uint32_t kTripRow = 24;  // at most 32: a short row's hits are one register
constexpr int kHitTrips = 8;  // divides 32; 4-clique R-MAT-20 4.13 -> 4.06 ms against four
template <int P>
__device__ __forceinline__ void hit_rows(const Staged& st, const TrieView& t, const RevView& r, uint32_t kb,
                                         uint32_t ke, const uint32_t* __restrict__ moff,
                                         uint32_t* __restrict__ mask, const CliqueShare& share) {
  const uint32_t lane = lane_id();
  const uint32_t step = r.dir == DIR_DOWN ? 0xffffffffu : 1u;  // from one candidate's element to the next's
  uint32_t next_lo = 0, next_hi = 0, next_src = 0;  // the next batch's rows, loaded a batch ahead
  if (kb + lane < ke) {
    next_lo = __ldg(r.rev_lo + kb + lane);
    next_hi = __ldg(r.rev_hi + kb + lane);
    next_src = __ldg(r.rev_src + kb + lane);
  }
  for (uint32_t k0 = kb; k0 < ke; k0 += 32) {
    const uint32_t k = k0 + lane;
    const uint32_t lo = next_lo, hi = next_hi, src = next_src;
    if (k + 32 < ke) {
      next_lo = __ldg(r.rev_lo + k + 32);
      next_hi = __ldg(r.rev_hi + k + 32);
      next_src = __ldg(r.rev_src + k + 32);
    }
    uint32_t len = 0, fe = 0;               // candidates; the element of the first one
    uint32_t skip = 0, base = 0, rs = 0;    // bit of the first candidate in the row's words, first word, stride
    if (k < ke) {
      const uint32_t d = staged_range(t, src).len;
      if (share.builds(src, d)) {
        const uint32_t W = (d + 31) >> 5;
        len = hi - lo;
        const uint32_t i = d - 1 - len;
        fe = r.dir == DIR_DOWN ? hi - 1 : lo;
        skip = (i & 31) + 1;
        const uint32_t q = i >> 5;
        base = __ldg(moff + src) + hits_block(q, W) + (i & 31);
        rs = hits_stride(q, W, d);
      }
    }
    const bool is_long = len >= kTripRow;
    if (__any_sync(kFull, is_long)) {
      const uint32_t end = skip + len;      // bits skip .. end - 1 of the row's words
      const uint32_t f0 = skip >> 5;        // a row at the end of its block has no candidate in its first word
      const uint32_t nw = is_long ? ((end + 31) >> 5) - f0 : 0u;
      const uint32_t incl = warp_incl_scan(nw);
      const uint32_t total = __shfl_sync(kFull, incl, 31);
      const uint32_t word0 = f0 - (incl - nw);       // trip x of the list is word x + word0 of its row
      const uint32_t elem0 = fe - step * skip;       // bit p of the row is element elem0 + step * p
      for (uint32_t t0 = 0; t0 < total; t0 += 32) {
        uint32_t mine = 0;
        for (uint32_t u0 = 0; u0 < 32 && t0 + u0 < total; u0 += kHitTrips) {
          uint32_t v[kHitTrips];
#pragma unroll
          for (int u = 0; u < kHitTrips; u++) {
            const uint32_t x = min(t0 + u0 + u, total - 1);
            const int j = __popc(__ballot_sync(kFull, incl <= x));
            const uint32_t ej = __shfl_sync(kFull, elem0, j), lj = __shfl_sync(kFull, end, j);
            const uint32_t p = 32 * (x + __shfl_sync(kFull, word0, j)) + lane;
            v[u] = __ldg(t.vals + (ej + step * min(p, lj - 1)));  // bits outside the row are masked off below
          }
#pragma unroll
          for (int u = 0; u < kHitTrips; u++) {
            const uint32_t b = __ballot_sync(kFull, hit<P>(st, v[u]));
            if (lane == u0 + u) mine = b;
          }
        }
        const uint32_t x = min(t0 + lane, total - 1);
        const uint32_t j = owner_lane(incl, x);
        const uint32_t w = x + __shfl_sync(kFull, word0, j);
        const uint32_t sj = __shfl_sync(kFull, skip, j), lj = __shfl_sync(kFull, end, j);
        const uint32_t bj = __shfl_sync(kFull, base, j), rj = __shfl_sync(kFull, rs, j);
        if (sj > 32 * w) mine &= 0xffffffffu << (sj - 32 * w);  // sj - 32 w < 32: the word holds a candidate
        if (lj < 32 * w + 32) mine &= 0xffffffffu >> (32 * w + 32 - lj);
        if (mine && t0 + lane < total) mask[bj + w * rj] = mine;
      }
      if (is_long) len = 0;
    }
    const uint32_t incl = warp_incl_scan(len);
    const uint32_t total = __shfl_sync(kFull, incl, 31);
    const uint32_t excl = incl - len;
    const uint32_t elem0 = fe - step * excl;  // flattened pair q of the row is element elem0 + step * q
    uint32_t acc = 0;                         // the lane's short row, bit c = candidate c
    for (uint32_t p = 0; p < total; p += 32 * kShortUnroll) {
      uint32_t w[kShortUnroll];
#pragma unroll
      for (int u = 0; u < kShortUnroll; u++) {
        const uint32_t q = min(p + 32 * u + lane, total - 1);
        const uint32_t j = owner_lane(incl, q);
        w[u] = __ldg(t.vals + (__shfl_sync(kFull, elem0, j) + step * q));
      }
#pragma unroll
      for (int u = 0; u < kShortUnroll; u++) {
        const uint32_t p0 = p + 32 * u;
        const uint32_t ball = __ballot_sync(kFull, hit<P>(st, w[u]));
        const uint32_t s = max(excl, p0), e = min(incl, p0 + 32);
        if (s < e) {  // the row's candidates s - excl .. e - excl - 1 are bits s - p0 .. of the ballot
          const uint32_t bits = (ball >> (s - p0)) & (0xffffffffu >> (32 - (e - s)));
          acc |= bits << (s - excl);
        }
      }
    }
    if (acc) {
      const uint64_t m = (uint64_t)acc << skip;
      if ((uint32_t)m) mask[base] = (uint32_t)m;
      if ((uint32_t)(m >> 32)) mask[base + rs] = (uint32_t)(m >> 32);
    }
  }
}

// hit_rows for a merged item: each row's candidates looked up in its own entry's
// list.  Short rows are flattened as there; a longer one (the item holds 1024
// candidates at most) runs a mask word at a time.
__device__ __forceinline__ void hit_merged(const TrieView& t, const RevView& r, uint32_t h0, uint32_t kb, uint32_t ke,
                                           const uint32_t* __restrict__ moff, uint32_t* __restrict__ mask,
                                           const CliqueShare& share) {
  const uint32_t lane = lane_id();
  const uint32_t step = r.dir == DIR_DOWN ? 0xffffffffu : 1u;
  const Merged m(t, r, h0);
  for (uint32_t k0 = kb; k0 < ke; k0 += 32) {
    const uint32_t k = k0 + lane;
    uint32_t len = 0, fe = 0, skip = 0, base = 0, rs = 0;
    if (k < ke) {
      const uint32_t src = __ldg(r.rev_src + k);
      const uint32_t d = staged_range(t, src).len;
      if (share.builds(src, d)) {
        const uint32_t lo = __ldg(r.rev_lo + k), hi = __ldg(r.rev_hi + k);
        const uint32_t W = (d + 31) >> 5;
        len = hi - lo;
        const uint32_t i = d - 1 - len, q = i >> 5;
        fe = r.dir == DIR_DOWN ? hi - 1 : lo;
        skip = (i & 31) + 1;
        base = __ldg(moff + src) + hits_block(q, W) + (i & 31);
        rs = hits_stride(q, W, d);
      }
    }
    const uint32_t e = m.entry(min(k, ke - 1));
    const uint32_t s0 = __shfl_sync(kFull, (uint32_t)m.s0, e), n = __shfl_sync(kFull, m.len, e);
    uint32_t rows = __ballot_sync(kFull, len > 32);
    while (rows) {
      const int j = __ffs(rows) - 1;
      rows &= rows - 1;
      const uint32_t sk = __shfl_sync(kFull, skip, j), end = sk + __shfl_sync(kFull, len, j);
      const uint32_t ej = __shfl_sync(kFull, fe, j) - step * sk, sj = __shfl_sync(kFull, s0, j);
      const uint32_t nj = __shfl_sync(kFull, n, j), bj = __shfl_sync(kFull, base, j), rj = __shfl_sync(kFull, rs, j);
      for (uint32_t w = 0; 32 * w < end; w++) {
        const uint32_t p = 32 * w + lane;
        const uint32_t b = __ballot_sync(kFull, p >= sk && p < end && list_has(t.vals, sj, nj, __ldg(t.vals + (ej + step * min(max(p, sk), end - 1)))));
        if (lane == 0 && b) mask[bj + w * rj] = b;
      }
    }
    if (len > 32) len = 0;
    const uint32_t incl = warp_incl_scan(len);
    const uint32_t total = __shfl_sync(kFull, incl, 31);
    const uint32_t excl = incl - len;
    const uint32_t elem0 = fe - step * excl;
    uint32_t acc = 0;
    for (uint32_t p = 0; p < total; p += 64) {
      uint32_t w[2], sj[2], nj[2];
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const uint32_t q = min(p + 32 * u + lane, total - 1);
        const uint32_t j = owner_lane(incl, q);
        w[u] = __ldg(t.vals + (__shfl_sync(kFull, elem0, j) + step * q));
        sj[u] = __shfl_sync(kFull, s0, j);
        nj[u] = __shfl_sync(kFull, n, j);
      }
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const uint32_t p0 = p + 32 * u;
        const uint32_t ball = __ballot_sync(kFull, list_has(t.vals, sj[u], nj[u], w[u]));
        const uint32_t s = max(excl, p0), x = min(incl, p0 + 32);
        if (s < x) acc |= ((ball >> (s - p0)) & (0xffffffffu >> (32 - (x - s)))) << (s - excl);
      }
    }
    if (acc) {
      const uint64_t bits = (uint64_t)acc << skip;
      if ((uint32_t)bits) mask[base] = (uint32_t)bits;
      if ((uint32_t)(bits >> 32)) mask[base + rs] = (uint32_t)(bits >> 32);
    }
  }
}

// kOne: as in triangle_kernel
template <bool kOne>
__global__ void EH_TRI_LAUNCH_BOUNDS hits_kernel(const __grid_constant__ TrieView t1,
                                                 const __grid_constant__ RevView r1,
                                                 const TrieView* __restrict__ views, const RevView* __restrict__ revs,
                                                 const Item* __restrict__ items,
                                                 const unsigned int* __restrict__ n_items_p, int cap_words,
                                                 unsigned int* __restrict__ queue, HitsView hv, float* records) {
  extern __shared__ uint32_t smem[];
  const uint32_t lane = lane_id();
  uint32_t* sm = smem + (size_t)(threadIdx.x >> 5) * cap_words;
  const uint32_t n_items = __ldg(n_items_p);
  for (;;) {
    uint32_t it = 0;
    if (lane == 0) it = atomicAdd(queue, 1u);
    it = __shfl_sync(kFull, it, 0);
    if (it >= n_items) break;
    const Item item = items[it];
    TrieView tg;
    RevView rg;
    if (!kOne) {
      tg = views[item.g];
      rg = revs[item.g];
    }
    const TrieView& t = kOne ? t1 : tg;
    const RevView& r = kOne ? r1 : rg;
    const uint32_t* moff = hv.moff + hv.gstart[item.g];
    long long t0 = 0;
    if (records && lane == 0) t0 = clock64();
    if (item.hb & kMerged) {
      hit_merged(t, r, item.hb & ~kMerged, item.kb, item.ke, moff, hv.mask, hv.share);
      continue;
    }
    Staged st;
    // block bitsets too by their elements: probed where they lie, 4-clique and lollipop of
    // a star of 2^16 leaves in forced block layout took 7.0 and 9.1 ms, so 3.7 and 2.9
    const int mode = stage_set(t, item.hb, sm, cap_words, st, !few_candidates(r, item), true);
    switch (mode) {
      case P_SBITS:
        hit_rows<P_SBITS>(st, t, r, item.kb, item.ke, moff, hv.mask, hv.share);
        break;
      case P_GBITS:
        hit_rows<P_GBITS>(st, t, r, item.kb, item.ke, moff, hv.mask, hv.share);
        break;
      case P_SLIST:
        hit_rows<P_SLIST>(st, t, r, item.kb, item.ke, moff, hv.mask, hv.share);
        break;
      case P_GLIST:
        hit_rows<P_GLIST>(st, t, r, item.kb, item.ke, moff, hv.mask, hv.share);
        break;
      case P_ZBITS:
        hit_rows<P_ZBITS>(st, t, r, item.kb, item.ke, moff, hv.mask, hv.share);
        break;
      default:
        hit_rows<P_GBLOCK>(st, t, r, item.kb, item.ke, moff, hv.mask, hv.share);
        break;
    }
    __syncwarp();  // the staged region is reused by the next item
    if (records && lane == 0)
      write_record(records + 8 * (size_t)it, t, r, item, mode, (float)(clock64() - t0));
  }
}

// graph of global head entry gh
__device__ __forceinline__ uint32_t hits_graph(const HitsView& hv, uint32_t gh) {
  uint32_t lo = 0, hi = hv.n_graphs;  // first graph starting above gh
  while (lo + 1 < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (hv.gstart[mid] <= gh) lo = mid; else hi = mid;
  }
  return lo;
}
// global head entry of unit u: the last one whose units start at or before u
__device__ __forceinline__ uint32_t hits_unit_head(const HitsView& hv, uint32_t u) {
  uint32_t lo = 0, hi = hv.heads;  // first entry with upre > u, less one
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(hv.upre + mid) <= u) lo = mid + 1; else hi = mid;
  }
  return lo - 1;
}
// head entry of unit u, at or after head entry a.  The next few are looked at
// one by one (neighbours mostly have units); entries without units can lie in
// hundreds of thousands between two that have some, so then by search (two
// Erdos-Renyi graphs of 2^18 nodes, whose 4-clique units lie at the low ids of
// each: 12.9 ms walking, one load after the other, 0.20 with the search).
__device__ __forceinline__ uint32_t hits_unit_next(const HitsView& hv, uint32_t a, uint32_t u) {
  for (uint32_t end = a + 8; a < end; a++)  // unit u exists, so some entry below hv.heads is found
    if (__ldg(hv.upre + a + 1) > u) return a;
  return hits_unit_head(hv, u);
}

// Work units of a head entry in the second pass.
// 4-clique: eight rows of a part of d > 32 elements; smaller parts are one row
// per lane and have no units.  Annotation: one unit per word column.
enum { HITS_CLIQUE = 0, HITS_ANNOT = 1, HITS_ROWS = 2 };
__device__ __forceinline__ uint64_t hits_units(uint64_t d, int use) {
  const uint64_t W = (d + 31) / 32;
  if (use == HITS_ANNOT) return d >= 2 ? W : 0;
  if (use == HITS_ROWS || d <= 32) return 0;
  return (d + 7) / 8;
}

// mask words and second-pass units of every head entry, none for those that only
// other ranks build; the sums over all entries, their longest part and the sum of
// their hits_work, and the sums over the entries built here
__global__ void hits_size_kernel(TrieView t, int use, CliqueShare share, uint32_t* __restrict__ words,
                                 uint32_t* __restrict__ units, unsigned long long* __restrict__ sums) {
  unsigned long long sw = 0, su = 0, work = 0, bw = 0, bu = 0;
  uint32_t most = 0;
  for (uint32_t a = blockIdx.x * blockDim.x + threadIdx.x; a < t.n_head; a += gridDim.x * blockDim.x) {
    const uint64_t d = staged_range(t, a).len;
    const uint64_t w = hits_words(d), u = hits_units(d, use);
    const bool built = share.builds(a, (uint32_t)d);
    words[a] = built ? (uint32_t)w : 0u;  // meaningful only while the sum stays below 2^32, which the host checks
    units[a] = built ? (uint32_t)u : 0u;
    sw += w;
    su += u;
    bw += built ? w : 0;
    bu += built ? u : 0;
    work += hits_work(d);
    most = max(most, (uint32_t)d);
  }
  sw = warp_sum(sw);
  su = warp_sum(su);
  work = warp_sum(work);
  bw = warp_sum(bw);
  bu = warp_sum(bu);
  if (lane_id() == 0) {
    if (sw) atomicAdd(sums, sw);
    if (su) atomicAdd(sums + 1, su);
    if (work) atomicAdd(sums + 3, work);
    if (bw) atomicAdd(sums + 4, bw);
    if (bu) atomicAdd(sums + 5, bu);
  }
  most = __reduce_max_sync(kFull, most);
  if (lane_id() == 0 && most) atomicMax(sums + 2, (unsigned long long)most);
}

// 4-cliques whose lowest vertex (highest, on a relation that goes down) has a
// part of 3 to 32 elements: the matrix is one word per row, a row per lane.
// Warps take `span` head entries at a time, at most 32: one after the other, so
// that fewer are better while there are warps for them (batch of one graph, us, at
// 32 / fewer / without masks: K_48 71 / 47 / 132, Erdos-Renyi of 1024 nodes and
// degree 32 75 / 51 / 50).
__global__ void __launch_bounds__(256) clique_small_kernel(const TrieView* __restrict__ views, HitsView hv,
                                                           uint32_t span, unsigned long long* __restrict__ total) {
  const uint32_t lane = lane_id();
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  unsigned long long acc = 0;
  uint32_t cur_g = 0;
  for (uint64_t h0 = (uint64_t)span * warp; h0 < hv.heads; h0 += (uint64_t)span * nwarps) {
    const uint32_t gh = (uint32_t)h0 + lane;
    uint32_t d = 0, mo = 0, g = 0;
    if (lane < span && gh < hv.heads) {
      g = hv.n_graphs > 1 ? hits_graph(hv, gh) : 0;
      const TrieView& t = views[g];
      const uint32_t a = gh - hv.gstart[g];
      d = staged_range(t, a).len;
      if (!hv.share.owns(a, d, 0)) d = 0;
      mo = __ldg(hv.moff + gh);
    }
    uint32_t todo = __ballot_sync(kFull, d >= 3 && d <= 32);
    while (todo) {
      const int j = __ffs(todo) - 1;
      todo &= todo - 1;
      const uint32_t dj = __shfl_sync(kFull, d, j), mj = __shfl_sync(kFull, mo, j), gj = __shfl_sync(kFull, g, j);
      const uint32_t row = lane < dj ? __ldg(hv.mask + mj + lane) : 0u;
      uint32_t set = __ballot_sync(kFull, row != 0);
      if (gj != cur_g) {
        acc = warp_sum(acc);
        if (lane == 0 && acc) atomicAdd(total + cur_g, acc);
        acc = 0;
        cur_g = gj;
      }
      uint32_t c = 0;
      while (set) {
        const int b = __ffs(set) - 1;
        set &= set - 1;
        const uint32_t rb = __shfl_sync(kFull, row, b);
        if ((row >> b) & 1u) c += __popc(row & rb);
      }
      acc += c;
    }
  }
  acc = warp_sum(acc);
  if (lane == 0 && acc) atomicAdd(total + cur_g, acc);
}

// parts of more words than this (2048 neighbours) are clique_wide_kernel's
constexpr uint32_t kSparseWords = 64;

// A unit of the 4-clique: the eight rows at `rows` of row block qi of the matrix m (W
// words wide, d elements) against the blocks q0, q0 + step, ... of later positions.  A
// function of its own, or its caller's state takes registers from the loop (4-clique
// R-MAT-20, ms, so / inlined: at eight blocks per SM 3.78 / -, at six 3.98 / 3.99, at
// four 3.93 / 3.96).
__device__ __noinline__ uint32_t clique_dense(const uint32_t* m, const uint32_t* rows, uint32_t ri, uint32_t qi,
                                                 uint32_t W, uint32_t d, uint32_t q0, uint32_t step) {
  const uint32_t lane = lane_id();
  // below 2^29: the masks of all entries are 2^31 words at most, which bounds the
  // sum of all d^2 by 2^37, and a lane's j, at most 2^13, add up to 8 d_j each
  uint32_t c = 0;
  for (uint32_t q = q0; q < W; q += step) {
    const uint4 ma = __ldg(reinterpret_cast<const uint4*>(rows + (q - qi) * ri));
    const uint4 mb = __ldg(reinterpret_cast<const uint4*>(rows + (q - qi) * ri + 4));
    if (!(ma.x | ma.y | ma.z | ma.w | mb.x | mb.y | mb.z | mb.w)) continue;
    // all ones where the lane's position j = 32 q + lane is a hit of the row
    const uint32_t on[8] = {0u - ((ma.x >> lane) & 1u), 0u - ((ma.y >> lane) & 1u), 0u - ((ma.z >> lane) & 1u),
                            0u - ((ma.w >> lane) & 1u), 0u - ((mb.x >> lane) & 1u), 0u - ((mb.y >> lane) & 1u),
                            0u - ((mb.z >> lane) & 1u), 0u - ((mb.w >> lane) & 1u)};
    const uint32_t rq = hits_stride(q, W, d);
    const uint32_t* jw = m + hits_block(q, W) + lane;
    const bool has = lane < rq;
#pragma unroll 2
    for (uint32_t k = q; k < W; k++) {
      const uint32_t y = has ? __ldg(jw + (k - q) * rq) : 0u;
      const uint4 xa = __ldg(reinterpret_cast<const uint4*>(rows + (k - qi) * ri));
      const uint4 xb = __ldg(reinterpret_cast<const uint4*>(rows + (k - qi) * ri + 4));
      c += __popc(xa.x & y & on[0]) + __popc(xa.y & y & on[1]) + __popc(xa.z & y & on[2]) +
           __popc(xa.w & y & on[3]) + __popc(xb.x & y & on[4]) + __popc(xb.y & y & on[5]) +
           __popc(xb.z & y & on[6]) + __popc(xb.w & y & on[7]);
    }
  }
  return c;
}

// 4-cliques of the larger parts.  A unit is eight consecutive rows i of one
// matrix.  For a block q of 32 later positions j, each lane holds the row of
// one j and ANDs its words with the same words of the eight rows, of each row
// i whose bit j is set.  Row j's word is one line per warp and serves all eight
// rows, whose own words are two 16-byte loads, the same for all lanes; that
// leaves AND, popcount and add per (i, j word) and makes the popcounts (16
// lanes per clock) the bound.  A warp takes `grab` units in a row, the four of one
// row block where there are units enough: its L1 then holds the matrix.  Where there
// are fewer than warps, `slices` warps share a unit, each every so many of its blocks
// q (all four units of a block on one warp always, kernels, ms: star of 2^11 leaves
// 0.54, so 0.09, without masks 0.04; R-MAT-13 by its own ids 1.25 -> 0.25).
template <bool kSlices>
__global__ void __launch_bounds__(256, 8) clique_big_kernel(const TrieView* __restrict__ views, HitsView hv,
                                                         uint32_t n_units, uint32_t grab, uint32_t slices,
                                                         unsigned int* __restrict__ queue,
                                                         unsigned long long* __restrict__ total) {
  const uint32_t lane = lane_id();
  unsigned long long acc = 0;
  uint32_t cur_g = 0;
  for (;;) {
    uint32_t x0 = 0;
    if (lane == 0) x0 = atomicAdd(queue, grab);
    x0 = __shfl_sync(kFull, x0, 0);
    const uint32_t u0 = kSlices ? x0 / slices : x0;
    const uint32_t slice = kSlices ? x0 - u0 * slices : 0;
    if (u0 >= n_units) break;
    const uint32_t u1 = min(u0 + grab, n_units);
    uint32_t gh = hits_unit_head(hv, u0);
    for (uint32_t u = u0; u < u1; u++) {
      gh = hits_unit_next(hv, gh, u);
      const uint32_t g = hv.n_graphs > 1 ? hits_graph(hv, gh) : 0;
      if (g != cur_g) {
        acc = warp_sum(acc);
        if (lane == 0 && acc) atomicAdd(total + cur_g, acc);
        acc = 0;
        cur_g = g;
      }
      const uint32_t a = gh - hv.gstart[g], d = staged_range(views[g], a).len, W = (d + 31) >> 5;
      const uint32_t* m = hv.mask + __ldg(hv.moff + gh);
      const uint32_t i0 = 8 * (u - __ldg(hv.upre + gh)), qi = i0 >> 5, ri = hits_stride(qi, W, d);
      if (W > kSparseWords || !hv.share.owns(a, d, i0)) continue;
      const uint32_t* rows = m + hits_block(qi, W) + (i0 & 31);
      acc += clique_dense(m, rows, ri, qi, W, d, qi + slice, kSlices ? slices : 1);
    }
  }
  acc = warp_sum(acc);
  if (lane == 0 && acc) atomicAdd(total + cur_g, acc);
}

// 4-cliques of one row of a wide, nearly empty matrix: the non-zero words of row x of
// the unit, at most kRowWords of them at a time in `list` (word, bits), are ANDed with
// the same words of the row of each of its hits, every mw-th of them from `sub` on.
constexpr uint32_t kRowWords = 256;
__device__ __forceinline__ unsigned long long clique_sparse_row(const uint32_t* m, const uint32_t* row, uint32_t ri,
                                                                uint32_t qi, uint32_t W, uint32_t d, uint32_t sub,
                                                                uint32_t mw, uint2* list) {
  const uint32_t lane = lane_id();
  unsigned long long acc = 0;
  for (uint32_t next = qi; next < W;) {
    uint32_t n = 0;
    __syncwarp();
    for (; next < W && n <= kRowWords - 32; next += 32) {
      const uint32_t q = next + lane;
      const uint32_t w = q < W ? __ldg(row + (q - qi) * ri) : 0u;
      const uint32_t set = __ballot_sync(kFull, w != 0);
      if (w) list[n + __popc(set & lanemask_lt())] = make_uint2(q, w);
      n += __popc(set);
    }
    __syncwarp();
    if (!n) continue;
    uint32_t first = 0, hit = 0;  // first word of the list at or after the hit's; hits so far
    for (uint32_t q0 = qi; q0 < next; q0 += 32) {
      const uint32_t q = q0 + lane;
      const uint32_t w = q < W ? __ldg(row + (q - qi) * ri) : 0u;
      for (uint32_t set = __ballot_sync(kFull, w != 0); set; set &= set - 1) {
        const uint32_t qj = q0 + __ffs(set) - 1;
        while (first < n && list[first].x < qj) first++;
        const uint32_t rj = hits_stride(qj, W, d);
        const uint32_t* jw = m + hits_block(qj, W);
        for (uint32_t bits = __shfl_sync(kFull, w, qj - q0); bits; bits &= bits - 1) {
          if (hit++ % mw != sub) continue;
          const uint32_t* jr = jw + (__ffs(bits) - 1);
          uint32_t c = 0;
          for (uint32_t e = first + lane; e < n; e += 32) c += __popc(list[e].y & __ldg(jr + (list[e].x - qj) * rj));
          acc += c;
        }
      }
    }
  }
  return acc;
}

// 4-cliques of parts of more than kSparseWords words (ids not in degree order: a hub
// next to many).  One unit's AND can be millions of steps there, and its matrix nearly
// empty.  The warps of a block share a unit.  Each first weighs one of the eight rows:
// where the words of their hits' rows are few against the words to AND (32 scattered
// words against a step of three lines for eight rows, weighed 16 to 1) a warp takes one
// row by its non-zero words, else the warps take the blocks q in turn.
// Units of more than kHeavySteps steps go to a list that blocks work off in
// kHeavySlices pieces once they have seen their own units.  Nobody waits: a block
// leaves when it finds the list worked off or its next entry not yet written, and
// whoever is still writing one works the list off after that.
// (4-clique, kernels, ms, without masks / a warp per unit, sparse ones by pairs of at
// most 256 hits / so: Chung-Lu 2^20 of exponent 2.6 by its own ids 52 / 307 / 9.4, 2^15
// of 2.1 63 / 27 / 1.5, R-MAT-16 by its own ids 140 / 31 / 5.3, star of 2^17 leaves with
// 2^20 rows among them 32 / 15 / 13.8.  Heavy units shared by up to 17 blocks that each
// weigh them instead of the list: the star 110.)
constexpr uint32_t kHeavySteps = 16384, kHeavySlices = 32, kHeavySparse = 0x80000000u, kHeavyNone = 0xffffffffu;
struct HeavyUnits {
  unsigned int* count;  // [2] entries, pieces taken
  unsigned int* unit;   // [cap] unit, with kHeavySparse if it runs by its rows' words; kHeavyNone: not written
  uint32_t cap;
};
__global__ void __launch_bounds__(256, 4) clique_wide_kernel(const TrieView* __restrict__ views, HitsView hv,
                                                             uint32_t n_units, HeavyUnits heavy,
                                                             unsigned long long* __restrict__ total) {
  __shared__ uint2 s_list[8][kRowWords];
  __shared__ uint32_t s_unit[256];  // the wide units among the block's 256
  __shared__ uint32_t s_hits[8], s_words[8], s_steps[8];
  __shared__ unsigned int s_n;
  const uint32_t lane = lane_id(), wid = threadIdx.x >> 5;
  // slice s of S of unit u; weigh: decide how, and whether it is for the list
  auto run = [&](uint32_t u, bool weigh, bool sparse, uint32_t s, uint32_t S) {
    const uint32_t gh = hits_unit_head(hv, u);
    const uint32_t g = hv.n_graphs > 1 ? hits_graph(hv, gh) : 0, a = gh - hv.gstart[g];
    const uint32_t d = staged_range(views[g], a).len, W = (d + 31) >> 5;
    const uint32_t* m = hv.mask + __ldg(hv.moff + gh);
    const uint32_t i0 = 8 * (u - __ldg(hv.upre + gh)), qi = i0 >> 5, ri = hits_stride(qi, W, d);
    const uint32_t* rows = m + hits_block(qi, W) + (i0 & 31);
    if (weigh) {
      uint32_t h = 0, nz = 0, steps = 0;  // steps: of an AND of this row alone
      for (uint32_t q = qi + lane; q < W; q += 32) {
        const uint32_t w = __ldg(rows + wid + (q - qi) * ri);
        if (w) {
          h += __popc(w);
          nz++;
          steps += W - q;
        }
      }
      h = __reduce_add_sync(kFull, h);
      nz = __reduce_add_sync(kFull, nz);
      steps = __reduce_add_sync(kFull, steps);
      if (lane == 0) {
        s_hits[wid] = h;
        s_words[wid] = nz;
        s_steps[wid] = steps;
      }
      __syncthreads();
      uint64_t pairs = 0;  // (hit, word) pairs, at least one step of 32 per hit
      const float full = 0.5f * (float)(W - qi) * (float)(W - qi + 1);
      float empty = 1.f;  // share of the steps that no row needs, if their words lie independently
#pragma unroll
      for (int r = 0; r < 8; r++) {
        pairs += (uint64_t)s_hits[r] * (s_words[r] + 32);
        empty *= 1.f - (float)s_steps[r] / full;
      }
      if (!pairs) return;  // the same on every thread, as all that follows from these numbers
      const float dense = full * (1.f - empty);
      sparse = (float)pairs < 4.f * dense;
      if ((sparse ? (float)pairs / 64.f : dense) > (float)kHeavySteps) {
        if (threadIdx.x == 0) {
          const uint32_t i = atomicAdd(heavy.count, 1u);
          if (i < heavy.cap) atomicExch(heavy.unit + i, sparse ? u | kHeavySparse : u);
          s_n = i < heavy.cap;  // the block's units are counted out already
        }
        __syncthreads();
        if (s_n) return;
      }
    }
    unsigned long long acc;
    if (sparse) acc = clique_sparse_row(m, rows + wid, ri, qi, W, d, s, S, s_list[wid]);
    else acc = clique_dense(m, rows, ri, qi, W, d, qi + 8 * s + wid, 8 * S);
    acc = warp_sum(acc);
    if (lane == 0 && acc) atomicAdd(total + g, acc);
  };
  for (uint64_t base = 0; base < n_units; base += 256ull * gridDim.x) {  // the same on every thread
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    const uint64_t u = base + (uint64_t)threadIdx.x * gridDim.x + blockIdx.x;
    if (u < n_units) {
      const uint32_t gh = hits_unit_head(hv, (uint32_t)u);
      const uint32_t g = hv.n_graphs > 1 ? hits_graph(hv, gh) : 0, a = gh - hv.gstart[g];
      const uint32_t d = staged_range(views[g], a).len;
      if (d > 32 * kSparseWords && hv.share.owns(a, d, 8 * ((uint32_t)u - __ldg(hv.upre + gh))))
        s_unit[atomicAdd(&s_n, 1u)] = (uint32_t)u;
    }
    __syncthreads();
    const uint32_t n = s_n;
    for (uint32_t x = 0; x < n; x++) {
      run(s_unit[x], true, false, 0, 1);
      __syncthreads();  // the rows' numbers are the next unit's
    }
    __syncthreads();  // everybody has seen n
  }
  for (;;) {
    if (threadIdx.x == 0) {
      s_n = 0;
      unsigned int piece = atomicAdd(heavy.count + 1, 0u);
      while (piece / kHeavySlices < heavy.cap) {
        const unsigned int code = atomicAdd(heavy.unit + piece / kHeavySlices, 0u);
        if (code == kHeavyNone) break;
        const unsigned int seen = atomicCAS(heavy.count + 1, piece, piece + 1);
        if (seen == piece) {
          s_n = 1;
          s_unit[0] = code;
          s_unit[1] = piece % kHeavySlices;
          break;
        }
        piece = seen;  // another block took it: the next one
      }
    }
    __syncthreads();
    if (!s_n) break;
    run(s_unit[0] & ~kHeavySparse, false, (s_unit[0] & kHeavySparse) != 0, s_unit[1], kHeavySlices);
    __syncthreads();
  }
}

// 32 x 32 bits, row r in lane r's word -> column c in lane c's word
__device__ __forceinline__ uint32_t transpose32(uint32_t x) {
  const uint32_t lane = lane_id();
  uint32_t m = 0x0000ffffu;
#pragma unroll
  for (int s = 16; s; s >>= 1) {
    const uint32_t y = __shfl_xor_sync(kFull, x, s);
    x = (lane & s) ? ((x & ~m) | ((y >> s) & m)) : ((x & m) | ((y & m) << s));
    m ^= m << (s >> 1);
  }
  return x;
}

// Annotation of a symmetric relation: every undirected triangle a < b < w
// found once adds 2 (its two orderings) to T of each of its three vertices.
// Unit k of a part is its word column k: the column sums of block column k
// (how often position j is the third vertex) and the row sums of block k (how
// often it is the second), one addition to T per element, and the row sums
// once more to T[a].
// The largest sets are in most matrices, and in a relation in degree order they
// are the last head entries, neighbours in T: their additions would queue up on
// a few L2 lines.  The last kHubs entries count in shared memory and are added
// to T once per block.
constexpr uint32_t kHubs = 4096;
// A unit of a part of W words is a chain of W + 1 loads and some.  kWide: the units of
// parts of more than kWidePart elements, each shared by up to the eight warps of a
// block; every unit's entry is looked up, a thread each.  Otherwise the units of the
// other parts.  (Split by column instead, the row sums of a wide part's first columns
// stayed on one warp: lollipop on a star of 2^16 leaves with 2^18 rows among them 10.5
// ms, so 2.9; without masks 6.6.  Kernels, ms, wide from 1024 / 4096 elements: star of
// 2^12 0.06 / 0.10, R-MAT-16 by its own ids 0.86 / 0.97, Chung-Lu 2^23, where the look-up
// is paid for little, 16.8 / 16.7, and from 512 17.6.)
constexpr uint32_t kWidePart = 4096;
constexpr uint32_t kWideShare = 64;  // words of a part per warp that shares its units

// slice s of S of unit k of entry a's matrix: the column sums of column k's tiles and
// the row sums of block k's words, added to T and the block's hubs
template <bool kWide>
__device__ __forceinline__ void annot_column(const TrieView& t, const HitsView& hv, uint32_t a, uint32_t k,
                                             uint32_t s, uint32_t S, uint32_t hub0, unsigned int* hub,
                                             unsigned long long* __restrict__ T) {
  const uint32_t lane = lane_id();
  const StagedRange pr = staged_range(t, a);
  const uint32_t d = pr.len, W = (d + 31) >> 5;
  const uint32_t* m = hv.mask + __ldg(hv.moff + a);
  uint32_t col = 0, row = 0;
  const uint32_t rk = hits_stride(k, W, d);
  const uint32_t* mk = m + hits_block(k, W) + lane;
  if (!kWide) {
    for (uint32_t q = 0; q <= k; q++) {
      const uint32_t rq = hits_stride(q, W, d);
      const uint32_t x = lane < rq ? __ldg(m + hits_block(q, W) + (k - q) * rq + lane) : 0u;
      if (__any_sync(kFull, x != 0)) col += __popc(transpose32(x));
    }
    if (lane < rk)
      for (uint32_t w = k; w < W; w++) row += __popc(__ldg(mk + (w - k) * rk));
  } else {
    for (uint32_t q0 = 4 * s; q0 <= k; q0 += 4 * S) {
      uint32_t x[4];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const uint32_t q = q0 + i;
        const uint32_t rq = hits_stride(q, W, d);
        x[i] = q <= k && lane < rq ? __ldg(m + hits_block(q, W) + (k - q) * rq + lane) : 0u;
      }
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (__any_sync(kFull, x[i] != 0)) col += __popc(transpose32(x[i]));
    }
    if (lane < rk)
#pragma unroll 4
      for (uint32_t w = k + s; w < W; w += S) row += __popc(__ldg(mk + (w - k) * rk));
  }
  if (col + row) {  // so the position is below d
    const uint32_t h = (uint32_t)__ldg(t.head_index + __ldg(t.vals + pr.s0 + 32 * k + lane));
    const uint32_t v = col + row;
    if (h < hub0) atomicAdd(T + h, 2ull * v);
    else if (atomicAdd(hub + (h - hub0), v) > 0xffffffffu - v) atomicAdd(T + h, 2ull << 32);  // wrapped
  }
  const uint32_t all = warp_sum(row);
  if (lane == 0 && all) atomicAdd(T + a, 2ull * all);
}

template <bool kWide>
__global__ void __launch_bounds__(256) annot_hits_kernel(TrieView t, HitsView hv, uint32_t n_units,
                                                         uint32_t run,
                                                         unsigned long long* __restrict__ T) {
  __shared__ unsigned int hub[kHubs];
  for (uint32_t i = threadIdx.x; i < kHubs; i += blockDim.x) hub[i] = 0;
  __syncthreads();
  const uint32_t hub0 = t.n_head > kHubs ? t.n_head - kHubs : 0;
  if (kWide) {
    __shared__ uint32_t s_a[256], s_k[256];  // the wide units among the block's 256
    __shared__ unsigned int s_n;
    const uint32_t wid = threadIdx.x >> 5;
    for (uint64_t base = 0; base < n_units; base += 256ull * gridDim.x) {  // the same on every thread
      if (threadIdx.x == 0) s_n = 0;
      __syncthreads();
      const uint64_t u = base + (uint64_t)threadIdx.x * gridDim.x + blockIdx.x;
      if (u < n_units) {
        const uint32_t a = hits_unit_head(hv, (uint32_t)u), k = (uint32_t)u - __ldg(hv.upre + a);
        if (staged_range(t, a).len > kWidePart) {
          const uint32_t i = atomicAdd(&s_n, 1u);
          s_a[i] = a;
          s_k[i] = k;
        }
      }
      __syncthreads();
      const uint32_t n = s_n;
      for (uint32_t i = 0; i < n; i++) {
        const uint32_t a = s_a[i];
        const uint32_t S = min(8u, 1 + (staged_range(t, a).len >> 5) / kWideShare), s = (wid + i) & 7;
        if (s < S) annot_column<true>(t, hv, a, s_k[i], s, S, hub0, hub, T);
      }
      __syncthreads();
    }
  } else {
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    // runs of consecutive units, so that few searches find the head entries,
    // spread over the warps, so that the long rows of a range of ids are too
    uint32_t a = 0;
    for (uint64_t u0 = (uint64_t)warp * run; u0 < n_units; u0 += (uint64_t)nwarps * run) {
      const uint32_t u1 = (uint32_t)min(u0 + run, (uint64_t)n_units);
      a = hits_unit_head(hv, (uint32_t)u0);
      for (uint32_t u = (uint32_t)u0; u < u1; u++) {
        a = hits_unit_next(hv, a, u);
        if (staged_range(t, a).len <= kWidePart)
          annot_column<false>(t, hv, a, u - __ldg(hv.upre + a), 0, 1, hub0, hub, T);
      }
    }
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < kHubs; i += blockDim.x)
    if (hub[i]) atomicAdd(T + hub0 + i, 2ull * hub[i]);
}

// rows: triangles per relation row e = (a, position i); a warp per head entry
// would starve on short parts, so a thread per row
__device__ __forceinline__ uint32_t hits_position(int dir, const StagedRange& pr, uint64_t e) {
  return dir == DIR_DOWN ? pr.len - 1 - (uint32_t)(e - pr.s0) : (uint32_t)(e - pr.s0);
}
__global__ void hits_row_count_kernel(TrieView t, int dir, HitsView hv, const uint32_t* __restrict__ seg,
                                      uint64_t* __restrict__ cnt) {
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < t.rows; e += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t a = seg[e];
    const StagedRange pr = staged_range(t, a);
    uint32_t c = 0;
    if (pr.len >= 2) {
      const uint32_t d = pr.len, W = (d + 31) >> 5, i = hits_position(dir, pr, e), q = i >> 5;
      const uint32_t rs = hits_stride(q, W, d);
      const uint32_t* row = hv.mask + __ldg(hv.moff + a) + hits_block(q, W) + (i & 31);
      for (uint32_t k = 0; k < W - q; k++) c += __popc(__ldg(row + k * rs));
    }
    cnt[e] = c;
  }
}
// a warp per relation row with triangles: the words that hold some, found 32 at
// a time, a lane per bit; the relation's rows and the elements of a part are in
// ascending order, so the triangles come out sorted by (a, b, c).  (All words one
// after the other, the call on a star of 2^16 leaves with 2^18 rows among them
// took 33.0 ms; so 7.1.)
__global__ void __launch_bounds__(256) hits_row_write_kernel(TrieView t, int dir, HitsView hv,
                                                             const uint32_t* __restrict__ seg,
                                                             const uint64_t* __restrict__ pos, uint64_t total,
                                                             int stride, uint32_t* __restrict__ oa, uint32_t* __restrict__ ob,
                                                             uint32_t* __restrict__ oc) {
  const uint32_t lane = lane_id();
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  for (uint64_t e0 = 32ull * warp; e0 < t.rows; e0 += 32ull * nwarps) {
    const uint64_t el = e0 + lane;
    uint64_t p = 0, n = 0;
    if (el < t.rows) {
      p = pos[el];
      n = (el + 1 < t.rows ? pos[el + 1] : total) - p;
    }
    uint32_t todo = __ballot_sync(kFull, n != 0);
    while (todo) {
      const int l = __ffs(todo) - 1;
      todo &= todo - 1;
      const uint64_t e = e0 + l;
      uint64_t out = __shfl_sync(kFull, p, l);
      const uint32_t a = __ldg(seg + e);
      const StagedRange pr = staged_range(t, a);
      const uint32_t d = pr.len, W = (d + 31) >> 5, i = hits_position(dir, pr, e), q = i >> 5;
      const uint32_t rs = hits_stride(q, W, d);
      const uint32_t* row = hv.mask + __ldg(hv.moff + a) + hits_block(q, W) + (i & 31);
      const uint32_t va = __ldg(t.head + a), vb = __ldg(t.vals + e);
      for (uint32_t k0 = 0; k0 < W - q; k0 += 32) {
        // ascending elements: positions descend on a relation that goes down
        const uint32_t kl = dir == DIR_DOWN ? W - q - 1 - (k0 + lane) : k0 + lane;
        const uint32_t word = k0 + lane < W - q ? __ldg(row + kl * rs) : 0u;
        for (uint32_t words = __ballot_sync(kFull, word != 0); words; words &= words - 1) {
          const int j = __ffs(words) - 1;
          const uint32_t k = __shfl_sync(kFull, kl, j);
          uint32_t x = __shfl_sync(kFull, word, j);
          if (dir == DIR_DOWN) x = __brev(x);
          if ((x >> lane) & 1u) {
            const uint32_t bit = dir == DIR_DOWN ? 31 - lane : lane;
            const uint32_t p = 32 * (q + k) + bit;
            const uint64_t o = (out + __popc(x & lanemask_lt())) * stride;
            oa[o] = va;
            ob[o] = vb;
            oc[o] = __ldg(t.vals + pr.s0 + (dir == DIR_DOWN ? d - 1 - p : p));
          }
          out += __popc(x);
        }
      }
    }
  }
}

}  // namespace eh
