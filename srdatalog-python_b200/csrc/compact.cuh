// compact.cuh -- order-preserving stream compaction in two launches.
//
//   1. flag   : each block owns a contiguous chunk; every warp evaluates the
//               selector on 32 consecutive elements at a time and stores the
//               ballot as one flag word (bit l = element 32w + l); the block's
//               selected count goes to blk_counts;
//   2. write  : each block adds up the counts of the blocks before it (at
//               most 8 per SM: a few loads per thread, cheaper than a launch
//               that scans them), then walks its chunk a 2048-element tile
//               at a time; warp w takes the tile's elements
//               [256w, 256w + 256) in eight rounds of 32, so a round's output
//               positions are the running count plus the popcount of the
//               lower lanes of its flag word: loads and stores are coalesced.
//               The last block writes the total.
// No block waits on another, so nothing can spin.  Selectors provide
//   __device__ void block_setup(uint64_t begin, uint64_t end);  (all threads)
//   __device__ bool select(uint64_t i);
//   using value_type = ...;
//   __device__ value_type value(uint64_t i);        (what element i emits)
//   __device__ void store(uint64_t pos, value_type v);
#pragma once

#include "common.cuh"
#include "kernels.h"

namespace srdl {

constexpr int kCpThreads = 256;
constexpr int kCpWarps = kCpThreads / 32;
constexpr int kCpItems = 8;
constexpr int kCpTile = kCpThreads * kCpItems;
// The mark pass of the set difference: 16 keys a thread pay for a thread's
// search, and six blocks per SM (the shared memory's limit) fit one wave.  50M -
// 30M keys 426 us, 467 with 256 threads of 8 keys and four blocks, 485 with six.
constexpr int kDmThreads = 128;
constexpr int kDmItems = kCpTile / kDmThreads;

// Whether a set difference streams FULL (its merge path) or searches every key in
// it (its probe path).  Streaming costs both sides, a search one key, and few keys
// leave a merge's launches waiting on one another: the line is at 4.5 times the
// keys less 7M.  Merge / probe, us: 1M keys against 1M 40 / 33; 2M against 2M 50 /
// 45 and against 600k 39 / 41; 4M against 8M 78 / 85, 12M 96 / 91 and 16M 107 /
// 93; 10M against 30M 194 / 212 and 40M 222 / 225; 20M against 80M 398 / 435 and
// 100M 465 / 444; 50M against 25M 458 / 872 and 200M 953 / 1003.
__host__ __device__ inline bool dm_merges(uint64_t n, uint64_t n_full) {
  return 2 * (n_full + 7000000) <= 9 * n;
}

// Grid shape for n elements: every block owns `chunk` elements (a multiple
// of the tile), at most 8 blocks per SM, no empty blocks.
inline uint64_t cp_chunk(uint64_t n, int sms) {
  uint64_t tiles = (n + kCpTile - 1) / kCpTile;
  uint64_t cap = (uint64_t)sms * 8;
  uint64_t per = (tiles + cap - 1) / cap;
  return (per ? per : 1) * (uint64_t)kCpTile;
}
inline int cp_blocks(uint64_t n, uint64_t chunk) {
  uint64_t nb = (n + chunk - 1) / chunk;
  return nb ? (int)nb : 1;
}
// The same split with n known only on the device: nb blocks, whole tiles.
__device__ __forceinline__ uint64_t cp_even_chunk(uint64_t n, uint64_t nb) {
  const uint64_t tiles = (n + kCpTile - 1) / kCpTile;
  const uint64_t per = (tiles + nb - 1) / nb;
  return (per ? per : 1) * (uint64_t)kCpTile;
}
inline uint64_t cp_words(uint64_t n) { return (n + 31) / 32; }
inline size_t cp_scratch_bytes(uint64_t n) {
  // flag words + per-block counts (blocks <= 8 per SM; 256 SMs bound), and for
  // the set difference the merge-path cuts and HEAD positions of every tile
  // boundary (FULL at most 4.5 times the keys there), each piece padded to 256
  // bytes, plus alignment slack for the region itself
  const uint64_t mtiles = (n * 11 / 2 + kCpTile - 1) / kCpTile + 2;
  return ((cp_words(n) * 4 + 255) & ~uint64_t(255)) + (size_t)(256 * 8 + 1) * 4 + 3 * 256 +
         2 * ((mtiles * 8 + 255) & ~uint64_t(255)) + 256;
}

// With d_n (device loop), n is a capacity and the count is *d_n; chunk 0
// then means the even split of the true count over the grid.
template <class Sel>
__global__ void __launch_bounds__(kCpThreads) cp_flag_kernel(Sel sel, uint64_t n, uint64_t chunk,
                                                             uint32_t* flags, uint32_t* blk_counts,
                                                             const uint64_t* d_n) {
  __shared__ uint32_t sh[kCpThreads / 32 + 1];
  n = dev_size(n, d_n);
  chunk = dev_chunk(chunk, n, kCpTile);
  const uint64_t begin = (uint64_t)blockIdx.x * chunk;
  const uint64_t end = begin + chunk < n ? begin + chunk : n;
  const int lane = threadIdx.x & 31;
  sel.block_setup(begin, end);
  uint32_t cnt = 0;
  // chunk starts are multiples of 32, so each round of a warp is one flag word
  for (uint64_t w0 = begin + (threadIdx.x & ~31u); w0 < end; w0 += kCpThreads) {
    const uint64_t i = w0 + lane;
    const bool f = i < end && sel.select(i);
    const uint32_t m = __ballot_sync(kAllLanes, f);
    if (lane == 0) flags[w0 / 32] = m;
    cnt += f;
  }
  uint32_t tot;
  block_excl_scan(cnt, sh, &tot);
  if (threadIdx.x == 0) blk_counts[blockIdx.x] = tot;
}

template <class Sel>
__global__ void __launch_bounds__(kCpThreads) cp_write_kernel(Sel sel, uint64_t n, uint64_t chunk,
                                                              const uint32_t* __restrict__ flags,
                                                              const uint32_t* __restrict__ blk_counts,
                                                              uint64_t* d_total,
                                                              const uint64_t* d_n) {
  __shared__ uint32_t wtot[2][kCpWarps];
  __shared__ uint64_t sh[kCpWarps + 1];
  n = dev_size(n, d_n);
  chunk = dev_chunk(chunk, n, kCpTile);
  const uint64_t begin = (uint64_t)blockIdx.x * chunk;
  const uint64_t end = begin + chunk < n ? begin + chunk : n;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned lt = lanemask_lt();
  uint64_t base = block_prefix(blk_counts, blockIdx.x, sh);
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *d_total = base + blk_counts[blockIdx.x];
  int par = 0;
  for (uint64_t tile = begin; tile < end; tile += kCpTile, par ^= 1) {
    // lane r < 8 fetches the flag word of round r of this warp's 256 elements
    const uint64_t w0 = tile + (uint64_t)wid * (kCpItems * 32);
    const uint64_t wi = w0 + (uint64_t)lane * 32;
    const uint32_t my_word = (lane < kCpItems && wi < end) ? flags[wi / 32] : 0u;
    // the eight rounds' element loads are all issued before the first
    // store (coalesced either way; this keeps eight loads in flight)
    typename Sel::value_type v[kCpItems];
#pragma unroll
    for (int r = 0; r < kCpItems; r++) {
      const uint64_t i = w0 + (uint64_t)r * 32 + lane;
      if (i < end) v[r] = sel.value(i);
    }
    const uint32_t wcount = warp_sum((uint32_t)__popc(my_word));
    if (lane == 0) wtot[par][wid] = wcount;
    __syncthreads();
    uint64_t pos = base;
    uint32_t tile_total = 0;
#pragma unroll
    for (int w = 0; w < kCpWarps; w++) {
      const uint32_t c = wtot[par][w];
      pos += w < wid ? c : 0;
      tile_total += c;
    }
#pragma unroll
    for (int r = 0; r < kCpItems; r++) {
      const uint32_t m = __shfl_sync(kAllLanes, my_word, r);
      if ((m >> lane) & 1u) sel.store(pos + __popc(m & lt), v[r]);
      pos += __popc(m);
    }
    base += tile_total;
  }
}

// Runs the two launches; the selected count lands in *d_total.  With d_n,
// n is a capacity and the element count is *d_n (device loop).
template <class Sel>
void compact(const Launch& L, Sel sel, uint64_t n, uint64_t* d_total, Scratch& s,
             const uint64_t* d_n = nullptr) {
  if (n == 0) {
    SRDL_CUDA(cudaMemsetAsync(d_total, 0, sizeof(uint64_t), L.stream));
    return;
  }
  const uint64_t chunk = cp_chunk(n, L.num_sms);
  const int nb = cp_blocks(n, chunk);
  const uint64_t kchunk = d_n ? 0 : chunk;
  uint32_t* flags = s.take<uint32_t>(cp_words(n));
  uint32_t* counts = s.take<uint32_t>(nb);
  cp_flag_kernel<Sel><<<nb, kCpThreads, 0, L.stream>>>(sel, n, kchunk, flags, counts, d_n);
  cp_write_kernel<Sel><<<nb, kCpThreads, 0, L.stream>>>(sel, n, kchunk, flags, counts, d_total, d_n);
  SRDL_CUDA(cudaGetLastError());
  count_launches(2);
}

// Keeps a[i] when it differs from a[i-1] (optional) and is absent from the
// sorted unique arrays full[0..n_full) and head[0..n_head) (a Device2Level
// relation's two segments; head may be empty).  Keys are stored compressed
// as (hi << bits) | lo and are expanded to (hi << 32) | lo on output.
// PLAIN: the keys are whole (bits = 32) and distinct, known at compile time --
// the standalone set difference, whose mark pass is bound by instructions: 50M
// - 30M keys took 504 us, 553 when the pass treated them as the sort's.
template <typename K, bool PLAIN = false>
struct DedupDiffSel {
  const K* a;
  int bits;
  bool dedup;
  const uint64_t* full;
  uint64_t n_full;
  uint64_t* out;
  const uint64_t* head = nullptr;
  uint64_t n_head = 0;
  const uint64_t* d_n_full = nullptr;  // device loop: FULL's count on the device (n_full = capacity)
  uint64_t out_cap = ~0ull;             // device loop: room in `out`; a key past it raises *d_overflow
  unsigned int* d_overflow = nullptr;

  __device__ __forceinline__ uint64_t expand(K c) const {
    if (PLAIN || (sizeof(K) == 8 && bits == 32)) return (uint64_t)c;
    const uint64_t m = (1ull << bits) - 1;
    return (((uint64_t)c >> bits) << 32) | ((uint64_t)c & m);
  }
  __device__ void block_setup(uint64_t, uint64_t) {}
  // (without FULL and HEAD: compact_diff takes the paths below otherwise)
  __device__ __forceinline__ bool repeats(K before, K key) const { return !PLAIN && dedup && before == key; }
  __device__ bool select(uint64_t i) const { return !(i > 0 && repeats(a[i - 1], a[i])); }
  using value_type = uint64_t;
  __device__ uint64_t value(uint64_t i) const { return expand(a[i]); }
  __device__ void store(uint64_t pos, uint64_t v) const {
    if (pos < out_cap) out[pos] = v;
    else if (d_overflow) *d_overflow = 1u;
  }
};

// Device loop (d_n set): the merge path and the probe path are both in the
// graph and each kernel runs only when the counts on the device select its
// path.  The merge path streams all of FULL; the probe path costs a binary
// search in FULL per key and nothing else.
enum DiffPath : int { kPathAny = 0, kPathMerge = 1, kPathProbe = 2 };

template <typename K, bool PLAIN>
__device__ __forceinline__ bool diff_path_runs(int path, const DedupDiffSel<K, PLAIN>& sel, uint64_t n) {
  if (path == kPathAny) return true;
  return (path == kPathMerge) == dm_merges(n, sel.n_full);
}

// lower_bound of kDdKeys keys of one lane in a[0..n) (n > 0): the halvings are
// the same for every key, so the lane keeps kDdKeys loads in flight.
constexpr int kDdKeys = 8;
__device__ __forceinline__ void dd_lower_bounds(const uint64_t* __restrict__ a, uint64_t n,
                                                const uint64_t (&k)[kDdKeys], bool (&found)[kDdKeys]) {
  uint64_t p[kDdKeys];
#pragma unroll
  for (int q = 0; q < kDdKeys; q++) p[q] = 0;
  while (n > 1) {
    const uint64_t half = n >> 1;
#pragma unroll
    for (int q = 0; q < kDdKeys; q++)
      if (__ldg(a + p[q] + half) <= k[q]) p[q] += half;
    n -= half;
  }
#pragma unroll
  for (int q = 0; q < kDdKeys; q++) found[q] = __ldg(a + p[q]) == k[q];
}

// Probe path: flag words and per-block counts by one binary search per key in
// FULL (and HEAD).  A warp takes eight rounds of 32 consecutive keys at a
// time, one search per round and lane, all eight interleaved: a late
// iteration's few keys would otherwise pay eight searches of about 23
// dependent loads one after another.  Neighbouring lanes' keys are
// neighbours, so the last steps of a round's searches share lines.  30k keys
// against 8M: 50 us for the whole set difference, 103 us with eight searches
// one after another per thread.
template <typename K, bool PLAIN>
__global__ void __launch_bounds__(kCpThreads) dd_probe_kernel(DedupDiffSel<K, PLAIN> sel, uint64_t n, uint64_t chunk,
                                                              uint32_t* __restrict__ flags,
                                                              uint32_t* __restrict__ blk_counts,
                                                              const uint64_t* d_n, int path) {
  __shared__ uint32_t sh[kCpThreads / 32 + 1];
  sel.n_full = dev_size(sel.n_full, sel.d_n_full);
  n = dev_size(n, d_n);
  if (!diff_path_runs(path, sel, n)) return;
  chunk = dev_chunk(chunk, n, kCpTile);
  const uint64_t begin = (uint64_t)blockIdx.x * chunk;
  const uint64_t end = begin + chunk < n ? begin + chunk : n;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t cnt = 0;  // (lane 0: the warp's)
  for (uint64_t tile = begin; tile < end; tile += kCpTile) {
    const uint64_t w0 = tile + (uint64_t)wid * (kDdKeys * 32);
    uint64_t k[kDdKeys];
    bool keep[kDdKeys], hit[kDdKeys];
#pragma unroll
    for (int q = 0; q < kDdKeys; q++) {
      const uint64_t i = w0 + q * 32 + lane;
      const K c = i < end ? sel.a[i] : K(0);
      keep[q] = i < end && !(i > 0 && !PLAIN && sel.repeats(sel.a[i - 1], c));
      k[q] = sel.expand(c);
    }
    if (sel.n_full) {
      dd_lower_bounds(sel.full, sel.n_full, k, hit);
#pragma unroll
      for (int q = 0; q < kDdKeys; q++) keep[q] &= !hit[q];
    }
    if (sel.n_head) {
      dd_lower_bounds(sel.head, sel.n_head, k, hit);
#pragma unroll
      for (int q = 0; q < kDdKeys; q++) keep[q] &= !hit[q];
    }
#pragma unroll
    for (int q = 0; q < kDdKeys; q++) {
      const uint32_t m = __ballot_sync(kAllLanes, keep[q]);
      if (lane == 0 && w0 + q * 32 < end) flags[(w0 + q * 32) / 32] = m;
      cnt += __popc(m);
    }
  }
  uint32_t tot;
  block_excl_scan(lane == 0 ? cnt : 0u, sh, &tot);
  if (threadIdx.x == 0) blk_counts[blockIdx.x] = tot;
}

// ---- merge-path flag pass (FULL streamed once) ------------------------------
//
// The keys a (sorted, possibly repeating) and FULL (sorted, unique) are
// merged, FULL first on equal values, and the merged sequence is cut into
// tiles of kCpTile elements (one thread per tile boundary finds the cut by
// merge-path binary search, and the tile's start in HEAD).  Persistent blocks
// walk the tiles; the next tile's two slices are copied into the second
// shared buffer with cp.async while the current tile is merged, 16 merged
// elements per thread.  An a-key is kept iff it differs from the last FULL
// key taken at or before it (so it is not in FULL) and from the a-key before
// it (dedup); HEAD, when present, is probed per kept key within the tile's
// HEAD range.  Bits are OR-ed into the flag words (a tile's a-range does not
// start on a word boundary).

// Number of a-keys among the first `diag` merged elements.
template <typename K, bool PLAIN>
__device__ __forceinline__ uint64_t dm_path(const DedupDiffSel<K, PLAIN>& sel, uint64_t na,
                                            uint64_t diag) {
  uint64_t lo = diag > sel.n_full ? diag - sel.n_full : 0;
  uint64_t hi = diag < na ? diag : na;
  while (lo < hi) {
    const uint64_t mid = (lo + hi) >> 1;
    if (sel.expand(sel.a[mid]) < sel.full[diag - 1 - mid]) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// split[t] = a-keys among the first t*kCpTile merged elements; hpos[t] = the
// HEAD position of a[split[t]] (n_head past the last key).
template <typename K, bool PLAIN>
__global__ void dm_split_kernel(DedupDiffSel<K, PLAIN> sel, uint64_t na, uint64_t tiles,
                                uint64_t* __restrict__ split, uint64_t* __restrict__ hpos,
                                const uint64_t* d_n, int path) {
  const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  sel.n_full = dev_size(sel.n_full, sel.d_n_full);
  na = dev_size(na, d_n);
  if (!diff_path_runs(path, sel, na)) return;
  if (d_n) tiles = (na + sel.n_full + kCpTile - 1) / kCpTile;
  if (t > tiles) return;
  const uint64_t total = na + sel.n_full;
  const uint64_t diag = t * kCpTile < total ? t * kCpTile : total;
  const uint64_t i = dm_path(sel, na, diag);
  split[t] = i;
  if (hpos)
    hpos[t] = i < na ? lower_bound_u64(sel.head, 0, sel.n_head, sel.expand(sel.a[i])) : sel.n_head;
}

template <int BYTES>
__device__ __forceinline__ void cp_async_small(void* smem, const void* gmem) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(s), "l"(gmem), "n"(BYTES)
               : "memory");
}

// One merged tile's slices: la a-keys (K) at the start of the buffer, lf FULL
// keys after them at an 8-byte boundary; returns nothing, commits one group.
template <typename K, bool PLAIN>
__device__ __forceinline__ void dm_fetch(const DedupDiffSel<K, PLAIN>& sel, unsigned char* buf,
                                         uint64_t i0, uint32_t la, uint64_t j0, uint32_t lf) {
  K* da = reinterpret_cast<K*>(buf);
  uint64_t* df = reinterpret_cast<uint64_t*>(buf + ((la * sizeof(K) + 7) & ~size_t(7)));
  for (uint32_t k = threadIdx.x; k < la; k += kDmThreads) cp_async_small<sizeof(K)>(da + k, sel.a + i0 + k);
  for (uint32_t k = threadIdx.x; k < lf; k += kDmThreads) cp_async_small<8>(df + k, sel.full + j0 + k);
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}

template <typename K, bool PLAIN>
__global__ void __launch_bounds__(kDmThreads) dm_mark_kernel(DedupDiffSel<K, PLAIN> sel, uint64_t na,
                                                             uint64_t tiles,
                                                             const uint64_t* __restrict__ split,
                                                             const uint64_t* __restrict__ hpos,
                                                             uint32_t* __restrict__ flags,
                                                             const uint64_t* d_n, int path) {
  __shared__ __align__(16) unsigned char buf[2][(kCpTile + 1) * 8];
  __shared__ uint32_t sbits[kCpTile / 32 + 2];
  sel.n_full = dev_size(sel.n_full, sel.d_n_full);
  na = dev_size(na, d_n);
  if (!diff_path_runs(path, sel, na)) return;
  if (d_n) tiles = (na + sel.n_full + kCpTile - 1) / kCpTile;
  const uint64_t total = na + sel.n_full;
  auto bounds = [&](uint64_t t, uint64_t& i0, uint64_t& i1, uint64_t& j0, uint64_t& j1) {
    const uint64_t d0 = t * kCpTile;
    const uint64_t d1 = d0 + kCpTile < total ? d0 + kCpTile : total;
    i0 = split[t];
    i1 = split[t + 1];
    j0 = d0 - i0;
    j1 = d1 - i1;
  };
  uint64_t t = blockIdx.x;
  if (t >= tiles) return;
  uint64_t i0, i1, j0, j1;
  bounds(t, i0, i1, j0, j1);
  dm_fetch(sel, buf[0], i0, (uint32_t)(i1 - i0), j0, (uint32_t)(j1 - j0));
  int cur = 0;
  for (;;) {
    const uint64_t tn = t + gridDim.x;
    uint64_t ni0 = 0, ni1 = 0, nj0 = 0, nj1 = 0;
    if (tn < tiles) {
      bounds(tn, ni0, ni1, nj0, nj1);
      dm_fetch(sel, buf[cur ^ 1], ni0, (uint32_t)(ni1 - ni0), nj0, (uint32_t)(nj1 - nj0));
    }
    const uint32_t la = (uint32_t)(i1 - i0), lf = (uint32_t)(j1 - j0);
    const uint64_t w0 = i0 / 32;
    const uint32_t nwords = la ? (uint32_t)((i1 - 1) / 32 - w0 + 1) : 0;
    for (uint32_t k = threadIdx.x; k < nwords; k += kDmThreads) sbits[k] = 0;
    // values just before the tile (for the first element of thread 0's run)
    const uint64_t edge_a = i0 > 0 ? sel.expand(sel.a[i0 - 1]) : 0;
    const uint64_t edge_f = j0 > 0 ? sel.full[j0 - 1] : 0;
    uint64_t h0 = 0, h1 = 0;
    if (hpos) {
      h0 = hpos[t];
      h1 = hpos[t + 1] + 1;
      h1 = h1 < sel.n_head ? h1 : sel.n_head;
    }
    if (tn < tiles) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    else asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    const K* sa = reinterpret_cast<const K*>(buf[cur]);
    const uint64_t* sf =
        reinterpret_cast<const uint64_t*>(buf[cur] + ((la * sizeof(K) + 7) & ~size_t(7)));
    const uint32_t diag = threadIdx.x * kDmItems;
    if (diag < la + lf && la) {
      uint32_t lo = diag > lf ? diag - lf : 0, hi = diag < la ? diag : la;
      while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (sel.expand(sa[mid]) < sf[diag - 1 - mid]) lo = mid + 1;
        else hi = mid;
      }
      uint32_t ia = lo, jf = diag - lo;
      bool has_f = jf > 0 || j0 > 0;
      uint64_t last_f = jf > 0 ? sf[jf - 1] : edge_f;
      bool has_p = ia > 0 || i0 > 0;
      uint64_t prev = ia > 0 ? sel.expand(sa[ia - 1]) : edge_a;
      // this thread's a-keys are consecutive: their bits fit two flag words
      const uint64_t wbase = (i0 + ia) / 32;
      uint64_t mask = 0;
      // No branch and (8-byte keys) one load a step: a list that has run out
      // leaves a value that the other's bound overrules.
      const uint64_t* both = reinterpret_cast<const uint64_t*>(sa);  // (8-byte keys: sf follows them)
      uint64_t x = sel.expand(sa[ia]), f = sf[jf];
      bool known = has_f & (last_f == x);                             // x is in FULL
      bool again = !PLAIN & sel.dedup & has_p & (prev == x);          // x repeats the key before it
      const uint32_t sh = (uint32_t)(i0 - wbase * 32);                // i0 + ia - wbase * 32 < 64
#pragma unroll
      for (int q = 0; q < kDmItems; q++) {
        const bool take_a = (jf >= lf) | ((ia < la) & (x < f));
        bool keep = take_a & (ia < la) & !known & !again;
        if (!PLAIN && keep && h1 > h0) {
          const uint64_t g = lower_bound_u64(sel.head, h0, h1, x);
          keep = !(g < h1 && sel.head[g] == x);
        }
        if (keep) mask |= 1ull << (sh + ia);
        known = !take_a & (f == x);
        ia += take_a;
        jf += !take_a;
        if constexpr (sizeof(K) == 8) {
          const uint64_t next = both[min(take_a ? ia : la + jf, (uint32_t)kCpTile)];
          const uint64_t nx = take_a ? sel.expand(next) : x;
          again = !PLAIN & (take_a ? sel.dedup & (nx == x) : again);
          x = nx;
          f = take_a ? f : next;
        } else if (take_a) {
          const uint64_t nx = sel.expand(sa[ia]);
          again = sel.dedup & (nx == x);
          x = nx;
        } else {
          f = sf[jf];
        }
      }
      if ((uint32_t)mask) atomicOr(&sbits[wbase - w0], (uint32_t)mask);
      if (mask >> 32) atomicOr(&sbits[wbase + 1 - w0], (uint32_t)(mask >> 32));
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < nwords; k += kDmThreads)
      if (sbits[k]) atomicOr(&flags[w0 + k], sbits[k]);
    __syncthreads();
    if (tn >= tiles) break;
    t = tn;
    i0 = ni0;
    i1 = ni1;
    j0 = nj0;
    j1 = nj1;
    cur ^= 1;
  }
}

// Per-block selected counts of a flag-word array (blocks own `chunk` keys).
template <typename K, bool PLAIN>
static __global__ void __launch_bounds__(kCpThreads) cp_count_kernel(const uint32_t* __restrict__ flags,
                                                              uint64_t n, uint64_t chunk,
                                                              uint32_t* blk_counts,
                                                              DedupDiffSel<K, PLAIN> sel,
                                                              const uint64_t* d_n, int path) {
  __shared__ uint32_t sh[kCpThreads / 32 + 1];
  sel.n_full = dev_size(sel.n_full, sel.d_n_full);
  n = dev_size(n, d_n);
  if (!diff_path_runs(path, sel, n)) return;
  chunk = dev_chunk(chunk, n, kCpTile);
  const uint64_t begin = (uint64_t)blockIdx.x * chunk;
  const uint64_t end = begin + chunk < n ? begin + chunk : n;
  uint32_t c = 0;
  for (uint64_t w = begin / 32 + threadIdx.x; w < (end + 31) / 32; w += kCpThreads)
    c += __popc(flags[w]);
  uint32_t tot;
  block_excl_scan(c, sh, &tot);
  if (threadIdx.x == 0) blk_counts[blockIdx.x] = tot;
}

// compact() for DedupDiffSel with a FULL array: merge path or one search per key
// (dm_merges).
template <typename K, bool PLAIN>
void compact_diff(const Launch& L, DedupDiffSel<K, PLAIN> sel, uint64_t n, uint64_t* d_total, Scratch& s) {
  if (!sel.head || sel.n_head == 0) {
    sel.head = nullptr;
    sel.n_head = 0;
  }
  if (!sel.full) sel.n_full = 0;
  if ((sel.n_full == 0 && !sel.head) || n == 0) {
    compact(L, sel, n, d_total, s);
    return;
  }
  const uint64_t chunk = cp_chunk(n, L.num_sms);
  const int nb = cp_blocks(n, chunk);
  uint32_t* flags = s.take<uint32_t>(cp_words(n));
  uint32_t* counts = s.take<uint32_t>(nb);
  if (sel.n_full && dm_merges(n, sel.n_full)) {
    const uint64_t mtiles = (n + sel.n_full + kCpTile - 1) / kCpTile;
    SRDL_REQUIRE(mtiles < (1ull << 31), kErrCapacity, "set difference: too many rows");
    uint64_t* split = s.take<uint64_t>(mtiles + 1);
    uint64_t* mhpos = sel.head ? s.take<uint64_t>(mtiles + 1) : nullptr;
    SRDL_CUDA(cudaMemsetAsync(flags, 0, cp_words(n) * 4, L.stream));
    dm_split_kernel<K, PLAIN><<<(unsigned)((mtiles + 1 + 255) / 256), 256, 0, L.stream>>>(sel, n, mtiles, split, mhpos,
                                                                                  nullptr, kPathAny);
    const unsigned mgrid = (unsigned)std::min<uint64_t>(mtiles, (uint64_t)L.num_sms * 6);
    dm_mark_kernel<K, PLAIN><<<mgrid, kDmThreads, 0, L.stream>>>(sel, n, mtiles, split, mhpos, flags, nullptr, kPathAny);
    cp_count_kernel<K, PLAIN><<<nb, kCpThreads, 0, L.stream>>>(flags, n, chunk, counts, sel, nullptr, kPathAny);
    count_launches(3);
  } else {
    dd_probe_kernel<K, PLAIN><<<nb, kCpThreads, 0, L.stream>>>(sel, n, chunk, flags, counts, nullptr, kPathAny);
    count_launches(1);
  }
  cp_write_kernel<DedupDiffSel<K, PLAIN>><<<nb, kCpThreads, 0, L.stream>>>(sel, n, chunk, flags, counts, d_total, nullptr);
  SRDL_CUDA(cudaGetLastError());
  count_launches(1);
}

// compact_diff with the key count on the device (device loop): `cap` keys
// of room, *d_n of them present, FULL's count at sel.d_n_full (n_full its
// capacity).  Both the merge path and the probe path are launched; each kernel
// runs only when the counts on the device select its path (the host's rule),
// so no host decision depends on the counts.  Grids are sized for the
// capacities and each block derives its share of the true counts.
inline size_t diff_dev_extra_bytes(uint64_t cap, uint64_t full_cap) {
  return ((cap + full_cap) / kCpTile + 2) * 8 + 512;
}

template <typename K, bool PLAIN>
void compact_diff_dev(const Launch& L, DedupDiffSel<K, PLAIN> sel, uint64_t cap, const uint64_t* d_n,
                      uint64_t* d_total, Scratch& s) {
  sel.head = nullptr;
  sel.n_head = 0;
  if (!sel.full || !sel.d_n_full) {
    sel.full = nullptr;
    sel.n_full = 0;
    sel.d_n_full = nullptr;
    compact(L, sel, cap, d_total, s, d_n);
    return;
  }
  const uint64_t chunk = cp_chunk(cap, L.num_sms);
  const int nb = cp_blocks(cap, chunk);
  const uint64_t mtiles = (cap + sel.n_full + kCpTile - 1) / kCpTile;
  uint32_t* flags = s.take<uint32_t>(cp_words(cap));
  uint32_t* counts = s.take<uint32_t>(nb);
  uint64_t* split = s.take<uint64_t>(mtiles + 1);
  // merge path: the mark pass ORs its bits into zeroed flag words
  SRDL_CUDA(cudaMemsetAsync(flags, 0, cp_words(cap) * 4, L.stream));
  dm_split_kernel<K, PLAIN><<<(unsigned)((mtiles + 1 + 255) / 256), 256, 0, L.stream>>>(sel, cap, mtiles, split, nullptr,
                                                                                d_n, kPathMerge);
  const unsigned mgrid = (unsigned)std::min<uint64_t>(mtiles, (uint64_t)L.num_sms * 6);
  dm_mark_kernel<K, PLAIN><<<mgrid, kDmThreads, 0, L.stream>>>(sel, cap, mtiles, split, nullptr, flags, d_n, kPathMerge);
  cp_count_kernel<K, PLAIN><<<nb, kCpThreads, 0, L.stream>>>(flags, cap, 0, counts, sel, d_n, kPathMerge);
  // probe path
  dd_probe_kernel<K, PLAIN><<<nb, kCpThreads, 0, L.stream>>>(sel, cap, 0, flags, counts, d_n, kPathProbe);
  // either way: the ordered write of the kept keys
  cp_write_kernel<DedupDiffSel<K, PLAIN>><<<nb, kCpThreads, 0, L.stream>>>(sel, cap, 0, flags, counts, d_total, d_n);
  SRDL_CUDA(cudaGetLastError());
  count_launches(5);
}

// Distinct first-column values of a sorted key array.
struct RootSel {
  const uint64_t* keys;
  uint32_t* roots;
  __device__ void block_setup(uint64_t, uint64_t) {}
  __device__ bool select(uint64_t i) const {
    return i == 0 || (keys[i] >> 32) != (keys[i - 1] >> 32);
  }
  using value_type = uint32_t;
  __device__ uint32_t value(uint64_t i) const { return (uint32_t)(keys[i] >> 32); }
  __device__ void store(uint64_t pos, uint32_t v) const { roots[pos] = v; }
};

}  // namespace srdl
