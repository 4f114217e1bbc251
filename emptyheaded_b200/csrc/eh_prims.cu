// Device-wide primitives written for this engine: exclusive scan, LSD radix
// sort of 64-bit keys, unique, max.  They replace the reference's TBB sort
// (storage_engine/src/Trie.cpp:403-404) and its sequential run detection
// (Trie.cpp:192-224, 291-302) inside the trie build.
#include <algorithm>

#include "eh_common.cuh"

namespace eh {

// ================================================================== scan
// Three-phase scan: per-tile reduce, scan of tile sums (recursive), per-tile
// scan with the tile's offset.  Tile = 256 threads x 8 items.
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

template <typename T>
__device__ __forceinline__ T block_excl_scan(T v, T* warp_tot, T* total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  T inc = warp_incl_scan(v);
  if (lane == 31) warp_tot[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    T w = lane < (kScanThreads / 32) ? warp_tot[lane] : T(0);
    T wi = warp_incl_scan(w);
    if (lane < (kScanThreads / 32)) warp_tot[lane] = wi - w;
    if (lane == (kScanThreads / 32) - 1) *total = wi;
  }
  __syncthreads();
  return inc - v + warp_tot[wid];
}

template <typename T>
__global__ void scan_reduce_kernel(const T* __restrict__ in, uint64_t n, T* __restrict__ tile_sums) {
  __shared__ T warp_tot[kScanThreads / 32];
  const uint64_t base = (uint64_t)blockIdx.x * kScanTile;
  T s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    uint64_t i = base + (uint64_t)k * kScanThreads + threadIdx.x;
    if (i < n) s += in[i];
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) warp_tot[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    T w = threadIdx.x < (kScanThreads / 32) ? warp_tot[threadIdx.x] : T(0);
    w = warp_sum(w);
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = w;
  }
}

template <typename T>
__global__ void scan_tile_kernel(const T* __restrict__ in, T* __restrict__ out, uint64_t n,
                                 const T* __restrict__ tile_offsets, T* __restrict__ total_dev) {
  __shared__ T warp_tot[kScanThreads / 32];
  __shared__ T tot;
  const uint64_t base = (uint64_t)blockIdx.x * kScanTile + (uint64_t)threadIdx.x * kScanItems;
  T v[kScanItems];
  T s = 0;
  // a thread's eight values lie together: 16-byte accesses where both arrays allow
  const bool wide = base + kScanItems <= n && !((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15u);
  constexpr int kVec = 16 / sizeof(T);
  struct alignas(16) Vec {
    T x[kVec];
  };
  if (wide) {
#pragma unroll
    for (int k = 0; k < kScanItems; k += kVec) {
      const Vec q = *reinterpret_cast<const Vec*>(in + base + k);
#pragma unroll
      for (int j = 0; j < kVec; j++) v[k + j] = q.x[j];
    }
  } else {
#pragma unroll
    for (int k = 0; k < kScanItems; k++) v[k] = base + k < n ? in[base + k] : T(0);
  }
#pragma unroll
  for (int k = 0; k < kScanItems; k++) s += v[k];
  T ex = block_excl_scan(s, warp_tot, &tot);
  const T off = tile_offsets ? tile_offsets[blockIdx.x] : T(0);
  T run = off + ex;
  if (wide) {
#pragma unroll
    for (int k = 0; k < kScanItems; k += kVec) {
      Vec q;
#pragma unroll
      for (int j = 0; j < kVec; j++) {
        q.x[j] = run;
        run += v[k + j];
      }
      *reinterpret_cast<Vec*>(out + base + k) = q;
    }
  } else {
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
      if (base + k < n) out[base + k] = run;
      run += v[k];
    }
  }
  if (total_dev && blockIdx.x == gridDim.x - 1 && threadIdx.x == kScanThreads - 1) *total_dev = run;
}

template <typename T>
void exclusive_scan(const T* in, T* out, uint64_t n, T* total_dev, cudaStream_t s) {
  if (n == 0) {
    if (total_dev) EH_CUDA(cudaMemsetAsync(total_dev, 0, sizeof(T), s));
    return;
  }
  const uint64_t tiles = (n + kScanTile - 1) / kScanTile;
  if (tiles == 1) {
    scan_tile_kernel<T><<<1, kScanThreads, 0, s>>>(in, out, n, nullptr, total_dev);
    EH_CHECK_LAUNCH();
    return;
  }
  DevBuf<T> sums(tiles, s);
  scan_reduce_kernel<T><<<(unsigned)tiles, kScanThreads, 0, s>>>(in, n, sums.p);
  EH_CHECK_LAUNCH();
  exclusive_scan<T>(sums.p, sums.p, tiles, nullptr, s);
  scan_tile_kernel<T><<<(unsigned)tiles, kScanThreads, 0, s>>>(in, out, n, sums.p, total_dev);
  EH_CHECK_LAUNCH();
}
template void exclusive_scan<uint32_t>(const uint32_t*, uint32_t*, uint64_t, uint32_t*, cudaStream_t);
template void exclusive_scan<uint64_t>(const uint64_t*, uint64_t*, uint64_t, uint64_t*, cudaStream_t);

// Kernels exclusive_scan launches for n inputs.
uint32_t scan_launches(uint64_t n) {
  if (n == 0) return 0;
  const uint64_t tiles = (n + kScanTile - 1) / kScanTile;
  return tiles == 1 ? 1u : 2u + scan_launches(tiles);
}

// Tile-sum elements exclusive_scan_scratch needs for n inputs (all levels).
uint64_t scan_scratch_elems(uint64_t n) {
  uint64_t need = 0;
  while (n > (uint64_t)kScanTile) {
    n = (n + kScanTile - 1) / kScanTile;
    need += n;
  }
  return need;
}

// exclusive_scan with its tile sums in caller memory (scratch_elems >=
// scan_scratch_elems(n)): allocates nothing.
template <typename T>
void exclusive_scan_scratch(const T* in, T* out, uint64_t n, T* total_dev, T* scratch, uint64_t scratch_elems,
                            cudaStream_t s) {
  if (n == 0) {
    if (total_dev) EH_CUDA(cudaMemsetAsync(total_dev, 0, sizeof(T), s));
    return;
  }
  const uint64_t tiles = (n + kScanTile - 1) / kScanTile;
  if (tiles == 1) {
    scan_tile_kernel<T><<<1, kScanThreads, 0, s>>>(in, out, n, nullptr, total_dev);
    EH_CHECK_LAUNCH();
    return;
  }
  EH_REQUIRE(scratch_elems >= tiles, EH_ERR_INVALID, "scan scratch too small");
  T* sums = scratch;
  scan_reduce_kernel<T><<<(unsigned)tiles, kScanThreads, 0, s>>>(in, n, sums);
  EH_CHECK_LAUNCH();
  exclusive_scan_scratch<T>(sums, sums, tiles, nullptr, scratch + tiles, scratch_elems - tiles, s);
  scan_tile_kernel<T><<<(unsigned)tiles, kScanThreads, 0, s>>>(in, out, n, sums, total_dev);
  EH_CHECK_LAUNCH();
}
template void exclusive_scan_scratch<uint32_t>(const uint32_t*, uint32_t*, uint64_t, uint32_t*, uint32_t*, uint64_t,
                                               cudaStream_t);

// ============================================================ radix sort
// LSD, 8-bit digits.  One pass = histogram per tile (digit-major counters),
// exclusive scan of the counters, stable scatter.  A tile is 8 warps x 16
// rounds x 32 keys; each warp ranks its keys stably, the lanes of one digit
// found by eight ballots, against a warp-private digit histogram in shared
// memory.  The scatter waits (loads, shared memory) more than it computes, so
// it holds four blocks per SM: 64 registers, the ranks packed in 16 bits (16 M
// keys of 64 bits: 196 us a pass at 128 registers and two blocks, IPC 0.63).
constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortRounds = 16;
constexpr int kSortTile = kSortThreads * kSortRounds;  // 4096 keys
constexpr int kSortBlocks = 4;                         // per SM
constexpr int kRadix = 256;

template <typename K>
__global__ void __launch_bounds__(kSortThreads) radix_hist_kernel(const K* __restrict__ keys, uint64_t n,
                                                                  int shift, uint32_t* __restrict__ counts,
                                                                  uint32_t tiles) {
  __shared__ uint32_t h[kRadix];
  h[threadIdx.x] = 0;
  __syncthreads();
  const uint64_t base = (uint64_t)blockIdx.x * kSortTile;
#pragma unroll 4
  for (int r = 0; r < kSortRounds; r++) {
    uint64_t i = base + (uint64_t)r * kSortThreads + threadIdx.x;
    if (i < n) atomicAdd(&h[(keys[i] >> shift) & 0xff], 1u);
  }
  __syncthreads();
  counts[(uint64_t)threadIdx.x * tiles + blockIdx.x] = h[threadIdx.x];
}

// kVals: a uint32 payload travels with each key.  The tile's keys are first
// placed in digit order in shared memory (stable: tile digit start + the
// warp's offset within the digit + the key's rank in its warp), then written
// out in that order, so consecutive threads write consecutive slots of one
// digit's run (coalesced) instead of 256 scattered runs per round.  With
// write_keys = 0 only the payloads are written (the last pass of a sort whose
// caller reads the payloads alone).
// the lanes of `valid` with this lane's digit
__device__ __forceinline__ uint32_t digit_peers(uint32_t d, uint32_t valid) {
  uint32_t peers = valid;
#pragma unroll
  for (int b = 0; b < 8; b++) {
    const bool on = (d >> b) & 1u;
    const uint32_t v = __ballot_sync(kFull, on);
    peers &= on ? v : ~v;
  }
  return peers;
}

template <typename K, bool kVals>
__global__ void __launch_bounds__(kSortThreads, kSortBlocks) radix_scatter_kernel(const K* __restrict__ keys,
                                                                     K* __restrict__ out, uint64_t n,
                                                                     int shift,
                                                                     const uint32_t* __restrict__ offsets,
                                                                     uint32_t tiles,
                                                                     const uint32_t* __restrict__ vin,
                                                                     uint32_t* __restrict__ vout, int write_keys) {
  __shared__ uint32_t whist[kSortWarps][kRadix];
  __shared__ uint32_t tile_off[kRadix];
  __shared__ uint32_t tstart[kRadix];
  __shared__ uint32_t wtot[kSortWarps];
  extern __shared__ __align__(16) unsigned char sort_smem[];  // kSortTile keys, then (kVals) kSortTile payloads
  K* skeys = reinterpret_cast<K*>(sort_smem);
  uint32_t* svals = reinterpret_cast<uint32_t*>(skeys + kSortTile);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < kSortWarps * kRadix; i += kSortThreads) (&whist[0][0])[i] = 0;
  tile_off[threadIdx.x] = offsets[(uint64_t)threadIdx.x * tiles + blockIdx.x];
  __syncthreads();
  // warp w owns keys [base + w*512, base + (w+1)*512), round-major
  const uint64_t tbase = (uint64_t)blockIdx.x * kSortTile;
  const uint64_t wbase = tbase + (uint64_t)wid * (32 * kSortRounds);
  K k[kSortRounds];
  uint32_t pos[kSortRounds / 2];  // offsets among the warp's keys of the digit, 16 bits each
  const uint32_t lt = lanemask_lt();
#pragma unroll
  for (int r = 0; r < kSortRounds; r++) {
    const uint64_t i = wbase + (uint64_t)r * 32 + lane;
    k[r] = i < n ? keys[i] : 0;
  }
  const uint64_t left = n > wbase ? n - wbase : 0;
#pragma unroll
  for (int r = 0; r < kSortRounds; r++) {
    const uint32_t valid = left >= (uint64_t)(r + 1) * 32 ? kFull : left <= (uint64_t)r * 32 ? 0u : (1u << (left - r * 32)) - 1u;
    const bool in = (valid >> lane) & 1u;
    const uint32_t d = (uint32_t)((k[r] >> shift) & 0xff);
    const uint32_t peers = digit_peers(d, valid);
    const uint32_t rank = __popc(peers & lt);
    uint32_t basecnt = 0;
    if (in) basecnt = whist[wid][d];
    __syncwarp();
    if (in && rank == 0) whist[wid][d] = basecnt + __popc(peers);
    __syncwarp();
    const uint32_t p = basecnt + rank;
    pos[r / 2] = r & 1 ? pos[r / 2] | p << 16 : p;
  }
  __syncthreads();
  // per-digit exclusive prefix over warps (thread t owns digit t), and the
  // tile's digit starts (exclusive scan over digits)
  uint32_t run = 0;
#pragma unroll
  for (int w = 0; w < kSortWarps; w++) {
    const uint32_t c = whist[w][threadIdx.x];
    whist[w][threadIdx.x] = run;
    run += c;
  }
  const uint32_t inc = warp_incl_scan(run);
  if (lane == 31) wtot[wid] = inc;
  __syncthreads();
  uint32_t before = 0;
  for (int w = 0; w < wid; w++) before += wtot[w];
  tstart[threadIdx.x] = before + inc - run;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kSortRounds; r++) {
    const uint64_t i = wbase + (uint64_t)r * 32 + lane;
    if (i < n) {
      const uint32_t d = (uint32_t)((k[r] >> shift) & 0xff);
      const uint32_t li = tstart[d] + whist[wid][d] + ((pos[r / 2] >> (r & 1 ? 16 : 0)) & 0xffffu);
      skeys[li] = k[r];
      if (kVals) svals[li] = vin[i];
    }
  }
  __syncthreads();
  const uint32_t cnt = (uint32_t)min((uint64_t)kSortTile, n - tbase);
  for (uint32_t j = threadIdx.x; j < cnt; j += kSortThreads) {
    const K key = skeys[j];
    const uint32_t d = (uint32_t)((key >> shift) & 0xff);
    const uint32_t dst = tile_off[d] + (j - tstart[d]);
    if (write_keys) out[dst] = key;
    if (kVals) vout[dst] = svals[j];
  }
}

template <typename K>
static size_t scatter_smem(bool vals) {
  return (size_t)kSortTile * (sizeof(K) + (vals ? 4 : 0));
}

template <typename K>
static void set_scatter_smem() {
  static bool done = false;  // the staged scatter takes more than the default 48 KB
  if (done) return;
  EH_CUDA(cudaFuncSetAttribute(radix_scatter_kernel<K, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)scatter_smem<K>(true)));
  EH_CUDA(cudaFuncSetAttribute(radix_scatter_kernel<K, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)scatter_smem<K>(false)));
  done = true;
}

// LSD passes; with vals != nullptr a uint32 payload follows its key
// (stable).  copy_back: the sorted keys (and payloads) end in keys / vals;
// otherwise only the payloads are produced, in the buffer returned (vals or
// vtmp), and the keys are left unspecified.
template <typename K>
static uint32_t* radix_sort_impl(K* keys, K* tmp, uint32_t* vals, uint32_t* vtmp, uint64_t n, int bits,
                                 bool copy_back, cudaStream_t s) {
  if (n < 2) return vals;
  EH_REQUIRE(n < (1ull << 32), EH_ERR_UNSUPPORTED, "radix sort supports fewer than 2^32 keys");
  const uint32_t tiles = (uint32_t)((n + kSortTile - 1) / kSortTile);
  // the counters, then the tile sums of their scan: taken once for all passes (a
  // buffer per scan was freed, and waited for, twice a pass)
  const uint64_t n_counts = (uint64_t)kRadix * tiles, n_sums = scan_scratch_elems(n_counts);
  DevBuf<uint32_t> counts(n_counts + n_sums, s);
  set_scatter_smem<K>();
  K* src = keys;
  K* dst = tmp;
  uint32_t* vsrc = vals;
  uint32_t* vdst = vtmp;
  for (int shift = 0; shift < bits; shift += 8) {
    const int write_keys = copy_back || shift + 8 < bits;
    radix_hist_kernel<K><<<tiles, kSortThreads, 0, s>>>(src, n, shift, counts.p, tiles);
    EH_CHECK_LAUNCH();
    exclusive_scan_scratch<uint32_t>(counts.p, counts.p, n_counts, nullptr, counts.p + n_counts, n_sums, s);
    if (vals)
      radix_scatter_kernel<K, true><<<tiles, kSortThreads, scatter_smem<K>(true), s>>>(
          src, dst, n, shift, counts.p, tiles, vsrc, vdst, write_keys);
    else
      radix_scatter_kernel<K, false><<<tiles, kSortThreads, scatter_smem<K>(false), s>>>(
          src, dst, n, shift, counts.p, tiles, nullptr, nullptr, write_keys);
    EH_CHECK_LAUNCH();
    std::swap(src, dst);
    std::swap(vsrc, vdst);
  }
  if (copy_back && src != keys) {
    EH_CUDA(cudaMemcpyAsync(keys, src, n * sizeof(K), cudaMemcpyDeviceToDevice, s));
    if (vals) EH_CUDA(cudaMemcpyAsync(vals, vsrc, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
    return vals;
  }
  return vsrc;
}

void radix_sort_u64(uint64_t* keys, uint64_t* tmp, uint64_t n, int bits, cudaStream_t s) {
  radix_sort_impl<uint64_t>(keys, tmp, nullptr, nullptr, n, bits, true, s);
}

void radix_sort_kv(uint64_t* keys, uint64_t* ktmp, uint32_t* vals, uint32_t* vtmp, uint64_t n, int bits,
                   cudaStream_t s) {
  radix_sort_impl<uint64_t>(keys, ktmp, vals, vtmp, n, bits, true, s);
}

uint32_t* radix_sort_payload_u32(uint32_t* keys, uint32_t* ktmp, uint32_t* vals, uint32_t* vtmp, uint64_t n, int bits,
                                 cudaStream_t s) {
  EH_REQUIRE(bits >= 1 && bits <= 32, EH_ERR_INVALID, "32-bit keys sort on 1 to 32 bits");
  return radix_sort_impl<uint32_t>(keys, ktmp, vals, vtmp, n, bits, false, s);
}

// ================================================================ unique
// Two passes over the keys and a scan of the tiles' counts between them: no
// flag or position per key is stored.
__global__ void __launch_bounds__(kScanThreads) unique_count_kernel(const uint64_t* __restrict__ keys, uint64_t n,
                                                                    uint32_t* __restrict__ tiles) {
  __shared__ uint32_t tot[kScanThreads / 32];
  const uint64_t base = (uint64_t)blockIdx.x * kScanTile;
  uint32_t c = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    const uint64_t i = base + (uint64_t)k * kScanThreads + threadIdx.x;
    if (i < n) c += i == 0 || keys[i] != keys[i - 1];
  }
  c = warp_sum(c);
  if ((threadIdx.x & 31) == 0) tot[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kScanThreads / 32; w++) c += tot[w];
    tiles[blockIdx.x] = c;
  }
}
__global__ void __launch_bounds__(kScanThreads) unique_write_kernel(const uint64_t* __restrict__ keys, uint64_t n,
                                                                    const uint32_t* __restrict__ tiles,
                                                                    uint64_t* __restrict__ out) {
  // round-major: a warp's keys of a round are consecutive
  __shared__ uint32_t cnt[kScanItems][kScanThreads / 32];
  const uint64_t base = (uint64_t)blockIdx.x * kScanTile;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint64_t key[kScanItems];
  uint32_t first[kScanItems];
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    const uint64_t i = base + (uint64_t)k * kScanThreads + threadIdx.x;
    key[k] = i < n ? keys[i] : 0;
    first[k] = __ballot_sync(kFull, i < n && (i == 0 || key[k] != keys[i - 1]));
    if (lane == 0) cnt[k][wid] = __popc(first[k]);
  }
  __syncthreads();
  if (threadIdx.x < 32) {  // exclusive scan of the 64 counts in key order
    uint32_t* c = &cnt[0][0];
    static_assert(kScanItems * kScanThreads / 32 == 64, "two counts per lane");
    const uint32_t a = c[2 * lane], b = c[2 * lane + 1];
    const uint32_t incl = warp_incl_scan(a + b);
    c[2 * lane] = incl - a - b;
    c[2 * lane + 1] = incl - b;
  }
  __syncthreads();
  const uint64_t t0 = tiles[blockIdx.x];
#pragma unroll
  for (int k = 0; k < kScanItems; k++)
    if ((first[k] >> lane) & 1u) out[t0 + cnt[k][wid] + __popc(first[k] & lanemask_lt())] = key[k];
}

uint64_t unique_sorted_u64(const uint64_t* keys, uint64_t* out, uint64_t n, cudaStream_t s) {
  if (n == 0) return 0;
  const uint64_t tiles = (n + kScanTile - 1) / kScanTile;
  DevBuf<uint32_t> cnt(tiles + 1, s);
  unique_count_kernel<<<(unsigned)tiles, kScanThreads, 0, s>>>(keys, n, cnt.p);
  EH_CHECK_LAUNCH();
  exclusive_scan<uint32_t>(cnt.p, cnt.p, tiles, cnt.p + tiles, s);
  unique_write_kernel<<<(unsigned)tiles, kScanThreads, 0, s>>>(keys, n, cnt.p, out);
  EH_CHECK_LAUNCH();
  uint32_t h = 0;
  EH_CUDA(cudaMemcpyAsync(&h, cnt.p + tiles, 4, cudaMemcpyDeviceToHost, s));
  EH_CUDA(cudaStreamSynchronize(s));
  return h;
}

// =================================================================== max
__global__ void max_kernel(const uint32_t* __restrict__ a, uint64_t n, uint32_t* __restrict__ out) {
  uint32_t m = 0;
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (; i + 3 * step < n; i += 4 * step)  // four loads in flight
    m = max(m, max(max(a[i], a[i + step]), max(a[i + 2 * step], a[i + 3 * step])));
  for (; i < n; i += step) m = max(m, a[i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(kFull, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

uint32_t max_u32(const uint32_t* a, uint64_t n, cudaStream_t s) {
  DevBuf<uint32_t> out(1, s);
  EH_CUDA(cudaMemsetAsync(out.p, 0, 4, s));
  if (n) {
    max_kernel<<<std::min<uint64_t>(num_sms() * 8, (n + 255) / 256), 256, 0, s>>>(a, n, out.p);
    EH_CHECK_LAUNCH();
  }
  uint32_t h = 0;
  EH_CUDA(cudaMemcpyAsync(&h, out.p, 4, cudaMemcpyDeviceToHost, s));
  EH_CUDA(cudaStreamSynchronize(s));
  return h;
}

}  // namespace eh
