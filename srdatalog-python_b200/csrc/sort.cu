// sort.cu -- index build: LSD radix sort of packed keys + fused dedup / difference.
//
// Replaces rebuild_index_fn -> zip_sort_columns (thrust::sort on a zip
// iterator, a CUB merge sort: RT/gpu/sort.h:297-302) followed by
// deduplicate_aggregate_and_unique (RT/gpu/deduplication.h:178-258) and, for
// ComputeDeltaIndex, DSAI::set_difference_update
// (RT/gpu/device_sorted_array_index.ipp:966-1130).
//
// Design.  Datalog creates no values: every value of every relation comes
// from the loaded inputs (and rule constants), so the runtime knows a bound
// 2^bits on all values.  A two-column key (hi, lo) is compressed to
// (hi << bits) | lo -- 32 bits when 2*bits <= 32 -- and sorted with stable
// counting passes over digits of at most kRsAutoBits bits (or the caller's
// Launch::radix_bits).  Each pass is a histogram launch (shared-memory counters
// per block), a per-digit scan over the blocks, and a scatter launch in which
// every warp ranks its keys with one ballot per digit bit, the tile is staged
// in shared memory in digit order and written out coalesced; the first pass
// reads the caller's keys and packs them on the way.  No block ever waits on
// another.  The dedup (and optional "not in FULL" test) runs as one
// order-preserving compaction over the sorted keys that also expands them back
// to (hi << 32) | lo.  Up to kRsSmall keys take one launch of one block.
#include <atomic>
#include <type_traits>

#include "compact.cuh"
#include "kernels.h"

namespace srdl {

constexpr int kRsThreads = 512;
constexpr int kRsWarps = kRsThreads / 32;
constexpr int kRsItems = 16;                     // keys per thread and tile, at most
constexpr int kRsTile = kRsThreads * kRsItems;   // 8192 keys per tile, at most
constexpr int kRsMinChunk = 2048;                // keys a block takes, at least
constexpr int kRsMaxBits = 9;                    // widest digit there is a kernel for
constexpr int kRsBlocksPerSm = 2;                // resident blocks
// Widest digit when the caller names none: 100M keys of 42 bits take 3.99 ms in
// five passes of at most 9 bits; with digits of 8 bits the sixth pass made them
// 8% slower, and a 10-bit digit's counters leave one block per SM.
constexpr int kRsAutoBits = 9;

int value_bits(uint32_t max_value) {
  int b = 0;
  while (b < 32 && (uint64_t(max_value) >> b) != 0) b++;
  return b ? b : 1;
}

// A key of the caller's array, (hi << 32) | lo, in packed form.
template <typename K>
__device__ __forceinline__ K rs_packed(uint64_t k, int bits, bool swap) {
  uint64_t hi = k >> 32, lo = k & 0xffffffffull;
  if (swap) {
    const uint64_t t = hi;
    hi = lo;
    lo = t;
  }
  return (K)((hi << bits) | lo);
}

// Keys per block when nb blocks share n: an even split in multiples of 512 (the
// histogram's 16-byte loads start there), kRsMinChunk at least.
__host__ __device__ __forceinline__ uint64_t rs_chunk(uint64_t n, uint64_t nb) {
  const uint64_t c = ((n + nb - 1) / nb + 511) & ~uint64_t(511);
  return c < (uint64_t)kRsMinChunk ? (uint64_t)kRsMinChunk : c;
}

// Digit counts of every block's chunk, digit-major.  The first pass (FIRST)
// reads the caller's keys and packs them on the way.
template <typename K, bool FIRST>
__global__ void __launch_bounds__(kRsThreads) rs_hist(const void* __restrict__ in, uint64_t n, uint64_t chunk,
                                                      int shift, int nbins, uint32_t* __restrict__ counts,
                                                      const uint64_t* d_n, int bits, bool swap) {
  __shared__ uint32_t h[1 << kRsMaxBits];
  n = dev_size(n, d_n);
  if (d_n) chunk = rs_chunk(n, gridDim.x);
  for (int d = threadIdx.x; d < nbins; d += kRsThreads) h[d] = 0;
  __syncthreads();
  const uint64_t begin = (uint64_t)blockIdx.x * chunk;
  const uint64_t end = begin + chunk < n ? begin + chunk : n;
  const uint32_t mask = nbins - 1;
  if constexpr (FIRST) {
    // 8-byte loads: the caller's array is only that aligned
    const uint64_t* raw = static_cast<const uint64_t*>(in);
    uint64_t i = begin + threadIdx.x;
    for (; i + 3 * kRsThreads < end; i += 4 * kRsThreads) {
      uint64_t k[4];
#pragma unroll
      for (int q = 0; q < 4; q++) k[q] = __ldg(raw + i + q * kRsThreads);
#pragma unroll
      for (int q = 0; q < 4; q++)
        atomicAdd(&h[(uint32_t)(rs_packed<K>(k[q], bits, swap) >> shift) & mask], 1u);
    }
    for (; i < end; i += kRsThreads)
      atomicAdd(&h[(uint32_t)(rs_packed<K>(__ldg(raw + i), bits, swap) >> shift) & mask], 1u);
  } else {
    // 16-byte loads: the chunk starts a multiple of 512 keys into a 256-byte
    // aligned array; a ragged tail is read key by key.
    const K* keys = static_cast<const K*>(in);
    constexpr uint64_t kPer = 16 / sizeof(K);
    const uint64_t vend = begin < end ? begin + (end - begin) / kPer * kPer : begin;
    const uint4* vec = reinterpret_cast<const uint4*>(keys + begin);
    auto add = [&](const uint4& v) {
      if constexpr (sizeof(K) == 8) {
        const uint64_t k0 = ((uint64_t)v.y << 32) | v.x, k1 = ((uint64_t)v.w << 32) | v.z;
        atomicAdd(&h[(uint32_t)(k0 >> shift) & mask], 1u);
        atomicAdd(&h[(uint32_t)(k1 >> shift) & mask], 1u);
      } else {
        atomicAdd(&h[(v.x >> shift) & mask], 1u);
        atomicAdd(&h[(v.y >> shift) & mask], 1u);
        atomicAdd(&h[(v.z >> shift) & mask], 1u);
        atomicAdd(&h[(v.w >> shift) & mask], 1u);
      }
    };
    const uint64_t nv = begin < end ? (vend - begin) / kPer : 0;
    uint64_t q = threadIdx.x;
    for (; q + kRsThreads < nv; q += 2 * kRsThreads) {
      const uint4 v0 = __ldg(vec + q), v1 = __ldg(vec + q + kRsThreads);
      add(v0);
      add(v1);
    }
    if (q < nv) add(__ldg(vec + q));
    for (uint64_t i = vend + threadIdx.x; i < end; i += kRsThreads)
      atomicAdd(&h[(uint32_t)(keys[i] >> shift) & mask], 1u);
  }
  __syncthreads();
  for (int d = threadIdx.x; d < nbins; d += kRsThreads) counts[(uint64_t)d * gridDim.x + blockIdx.x] = h[d];
}

// Block d turns row d of the digit-major counters (one counter per
// histogram block) into exclusive offsets within the digit, in place, and
// writes the digit's total to digit_tot[d].
constexpr int kRsScanThreads = 256;

__global__ void __launch_bounds__(kRsScanThreads) rs_rowscan(uint32_t* c, int nb,
                                                             uint32_t* __restrict__ digit_tot) {
  __shared__ uint32_t sh[kRsScanThreads / 32 + 1];
  uint32_t* row = c + (uint64_t)blockIdx.x * nb;
  const int per = (nb + kRsScanThreads - 1) / kRsScanThreads;
  const int s = threadIdx.x * per, e = min(nb, s + per);
  uint32_t sum = 0;
  for (int i = s; i < e; i++) sum += row[i];
  uint32_t tot;
  uint32_t run = block_excl_scan(sum, sh, &tot);
  for (int i = s; i < e; i++) {
    uint32_t v = row[i];
    row[i] = run;
    run += v;
  }
  if (threadIdx.x == 0) digit_tot[blockIdx.x] = tot;
}

// Shared memory of a scatter block: the staged tile, a 16-bit counter per
// warp and digit, and per digit the next output position and its offset from
// the staged position.
template <typename K, int DB>
constexpr size_t rs_smem_bytes() {
  constexpr size_t bins = 1 << DB;
  return kRsTile * sizeof(K) + kRsWarps * (bins < 8 ? 16 : bins * 2) + 2 * (bins < 4 ? 16 : bins * 4);
}

// Lanes of the warp whose digit equals this lane's: one ballot per digit bit.
// Written in PTX, a predicated complement and an AND per bit: with the loop in C++
// a sort of 100M keys of 42 bits takes 4.59 ms (4.38 with the complement as an
// exclusive or) instead of 4.00.
template <int DB>
__device__ __forceinline__ unsigned rs_peers(uint32_t d) {
  unsigned peers = kAllLanes;
#pragma unroll
  for (int b = 0; b < DB; b++)
    asm volatile(
        "{\n"
        "  .reg .pred p;\n"
        "  .reg .b32 t;\n"
        "  setp.ne.u32 p, %1, 0;\n"
        "  vote.sync.ballot.b32 t, p, 0xffffffff;\n"
        "  @!p not.b32 t, t;\n"
        "  and.b32 %0, %0, t;\n"
        "}\n"
        : "+r"(peers)
        : "r"(d & (1u << b)));
  return peers;
}

// Stable rank of each lane's digit among the earlier keys of its warp with the
// same digit; counter[d] holds the warp's keys of digit d so far.  The highest
// lane of a digit stores the new count, which it knows from its own rank.
// (Setting lane bits in a shared match mask instead of the ballots takes fewer
// instructions and more shared-memory accesses: 4.20 ms for those 100M keys.)
template <int DB>
__device__ __forceinline__ uint32_t rs_rank(uint16_t* counter, uint32_t d, unsigned lt, unsigned gt) {
  const unsigned peers = rs_peers<DB>(d);
  const uint32_t rank = counter[d] + __popc(peers & lt);
  __syncwarp();
  if (!(peers & gt)) counter[d] = (uint16_t)(rank + 1);
  __syncwarp();
  return rank;
}

// One counting pass over this block's chunk, a tile of at most kRsTile keys at
// a time, for digits of DB bits.
//
// A warp owns 32 * rounds consecutive keys of the tile, 32 per round, held in
// registers, and ranks them with rs_rank.  Two digits' counters share a word:
// one thread per word turns the warps' counts into staged positions, one block
// scan orders the digits.  The keys are then staged in digit order and, while
// the next tile's keys are being loaded into the registers they left, written
// out in runs.  Full tiles of 16 keys per thread take a path without bounds
// checks.
//
// Bound: integer operations, which issue every other cycle, and shared-memory
// wavefronts (each about half used: two blocks of 16 warps share an SM);
// 16 keys per thread spread the per-digit work over 8192 keys and keep a tile's
// runs at 128 bytes for 9-bit digits.  100M keys of 42 bits: 0.58 ms per 9-bit
// pass, against 0.60 ms per 7-bit pass with 2048-key tiles and the ballots
// compiled from C++.  Tiles of 6144 keys with three blocks per SM, tiles of 4096
// with four, and rounds ranked four at a time were 7%, 8% and 3% slower.  Keys
// past the end are all ones: they rank behind every real key and are not
// written.
template <typename K, int DB, bool FIRST>
__global__ void __launch_bounds__(kRsThreads, 2) rs_scatter(const void* __restrict__ in, K* __restrict__ out,
                                                            uint64_t n, uint64_t chunk, int shift,
                                                            const uint32_t* __restrict__ offs,
                                                            const uint32_t* __restrict__ digit_tot,
                                                            const uint64_t* d_n, int bits, bool swap) {
  constexpr int nbins = 1 << DB;
  constexpr uint32_t mask = nbins - 1;
  constexpr int pairs = nbins / 2;                 // words holding two counters
  constexpr int stride = pairs < 4 ? 4 : pairs;    // words per warp
  extern __shared__ __align__(16) unsigned char rs_sm[];
  K* buf = reinterpret_cast<K*>(rs_sm);
  uint32_t* cnt = reinterpret_cast<uint32_t*>(rs_sm + kRsTile * sizeof(K));
  uint32_t* base = cnt + kRsWarps * stride;        // next global output position per digit
  uint32_t* gofs = base + (nbins < 4 ? 4 : nbins); // base minus the digit's start in the staged tile
  __shared__ uint32_t scan_sh[kRsWarps + 1];
  static_assert(pairs <= kRsThreads, "one thread per counter word");

  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  n = dev_size(n, d_n);
  if (d_n) chunk = rs_chunk(n, gridDim.x);
  const uint64_t begin = (uint64_t)blockIdx.x * chunk;
  const uint64_t end = begin + chunk < n ? begin + chunk : n;
  if (begin >= end) return;
  const uint32_t len = (uint32_t)(end - begin);
  const uint32_t ntiles = (len + kRsTile - 1) / kRsTile;
  // equal tiles: rounds <= kRsItems
  const int rounds = (int)((len + ntiles * kRsThreads - 1) / (ntiles * kRsThreads));
  const uint32_t tile_keys = (uint32_t)rounds * kRsThreads;

  K key[kRsItems];
  auto fetch = [&](uint64_t i) -> K {
    if constexpr (FIRST) return rs_packed<K>(__ldg(static_cast<const uint64_t*>(in) + i), bits, swap);
    else return __ldg(static_cast<const K*>(in) + i);
  };
  auto load = [&](uint64_t tile) {
    const uint64_t i0 = tile + (uint32_t)(wid * rounds * 32 + lane);
    if (rounds == kRsItems && tile + kRsTile <= end) {
#pragma unroll
      for (int r = 0; r < kRsItems; r++) key[r] = fetch(i0 + r * 32);
      return;
    }
#pragma unroll
    for (int r = 0; r < kRsItems; r++) {
      key[r] = ~K(0);
      if (r < rounds && i0 + r * 32 < end) key[r] = fetch(i0 + r * 32);
    }
  };
  load(begin);
  {
    // digit base = keys with a smaller digit; plus this block's offset in the digit
    const int t = threadIdx.x;
    const uint32_t t0 = t < pairs ? digit_tot[2 * t] : 0, t1 = t < pairs ? digit_tot[2 * t + 1] : 0;
    uint32_t all;
    const uint32_t db = block_excl_scan(t0 + t1, scan_sh, &all);
    if (t < pairs) {
      base[2 * t] = db + offs[(uint64_t)(2 * t) * gridDim.x + blockIdx.x];
      base[2 * t + 1] = db + t0 + offs[(uint64_t)(2 * t + 1) * gridDim.x + blockIdx.x];
    }
  }
  const unsigned lt = lanemask_lt(), gt = ~(lt | (1u << lane));
  uint32_t* my = cnt + wid * stride;
  uint16_t* my16 = reinterpret_cast<uint16_t*>(my);
  for (uint64_t tile = begin; tile < end; tile += tile_keys) {
    const uint32_t count = (uint32_t)(end - tile < tile_keys ? end - tile : tile_keys);
    for (int i = lane; i < stride; i += 32) my[i] = 0;
    __syncwarp();
    uint32_t rank[kRsItems / 2];  // two 16-bit ranks within the warp's digit run per word
#pragma unroll
    for (int r = 0; r < kRsItems; r++) {
      if (r < rounds) {
        const uint32_t rk = rs_rank<DB>(my16, (uint32_t)(key[r] >> shift) & mask, lt, gt);
        rank[r / 2] = r & 1 ? rank[r / 2] | (rk << 16) : rk;
      }
    }
    __syncthreads();
    // Per digit: staged start of each warp's run (tile start of the digit plus
    // the earlier warps' counts), and the global offset of the digit's run.
    {
      const int t = threadIdx.x;
      uint32_t run = 0;
      if (t < pairs) {
#pragma unroll
        for (int w = 0; w < kRsWarps; w++) {
          const uint32_t v = cnt[w * stride + t];
          cnt[w * stride + t] = run;
          run += v;  // (both halves stay below 2^16: a tile has 8192 keys)
        }
      }
      const uint32_t c0 = run & 0xffffu, c1 = run >> 16;
      uint32_t all;
      const uint32_t start = block_excl_scan(c0 + c1, scan_sh, &all);
      if (t < pairs) {
        const uint32_t b0 = base[2 * t], b1 = base[2 * t + 1];
        gofs[2 * t] = b0 - start;
        gofs[2 * t + 1] = b1 - (start + c0);
        base[2 * t] = b0 + c0;
        base[2 * t + 1] = b1 + c1;
        const uint32_t add = start | ((start + c0) << 16);
#pragma unroll
        for (int w = 0; w < kRsWarps; w++) cnt[w * stride + t] += add;
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kRsItems; r++) {
      if (r < rounds) {
        const uint32_t rk = r & 1 ? rank[r / 2] >> 16 : rank[r / 2] & 0xffffu;
        buf[my16[(uint32_t)(key[r] >> shift) & mask] + rk] = key[r];
      }
    }
    __syncthreads();
    if (tile + tile_keys < end) load(tile + tile_keys);
    // (the next tile's stores into buf and gofs come after its first barrier)
    if (count == kRsTile) {
#pragma unroll
      for (int q = 0; q < kRsItems; q++) {
        const K k = buf[threadIdx.x + q * kRsThreads];
        out[gofs[(uint32_t)(k >> shift) & mask] + (threadIdx.x + q * kRsThreads)] = k;
      }
    } else {
      for (uint32_t j = threadIdx.x; j < count; j += kRsThreads) {
        const K k = buf[j];
        out[gofs[(uint32_t)(k >> shift) & mask] + j] = k;
      }
    }
  }
}

// ---- at most kRsSmall keys: one block, one launch ----------------------------
//
// A small request's or a late iteration's tuples cost launches, not work: the
// passes above take three launches each whatever the count, about 3 us apiece.
// One block holds up to 16384 keys in shared memory, runs every counting pass
// there (8-bit digits, ranked by rs_rank), drops repeats and the keys
// found in FULL or HEAD (one interleaved binary search per key) and writes the
// rest in order.  Bound: one SM's issue slots; 5000 keys of 34 bits take 46 us
// with the count read back (109 us in 16 launches), 16,000 keys 71 us (95 us).
constexpr int kRsSmallThreads = 1024;
constexpr int kRsSmallWarps = kRsSmallThreads / 32;
constexpr uint64_t kRsSmall = (uint64_t)kRsSmallThreads * kRsItems;
static_assert(kRsSmall == kSortSmall, "one thread per kRsItems keys");
constexpr int kRsSmallBits = 8;
constexpr int kRsSmallPairs = 1 << (kRsSmallBits - 1);

template <typename K>
constexpr size_t rs_small_smem_bytes() {
  return kRsSmall * sizeof(K) + (size_t)kRsSmallWarps * kRsSmallPairs * 4;
}

template <typename K>
__global__ void __launch_bounds__(kRsSmallThreads, 1) rs_small_kernel(const uint64_t* in, uint32_t n, int bits,
                                                                      bool swap, int passes, DedupDiffSel<K> sel,
                                                                      uint64_t* d_nout) {
  extern __shared__ __align__(16) unsigned char rs_sm[];
  K* buf = reinterpret_cast<K*>(rs_sm);
  uint32_t* cnt = reinterpret_cast<uint32_t*>(rs_sm + kRsSmall * sizeof(K));
  __shared__ uint32_t scan_sh[kRsSmallWarps + 1];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned lt = lanemask_lt(), gt = ~(lt | (1u << lane));
  const int rounds = (int)((n + kRsSmallThreads - 1) / kRsSmallThreads);
  const uint32_t i0 = (uint32_t)(wid * rounds * 32 + lane);  // this lane's keys: i0, i0 + 32, ...
  uint32_t* my = cnt + wid * kRsSmallPairs;
  uint16_t* my16 = reinterpret_cast<uint16_t*>(my);
  K key[kRsItems];
#pragma unroll
  for (int r = 0; r < kRsItems; r++) {
    key[r] = ~K(0);  // behind every real key, in every pass
    if (r < rounds && i0 + r * 32 < n) key[r] = rs_packed<K>(in[i0 + r * 32], bits, swap);
  }
  const int total = 2 * bits;
  int shift = 0;
  for (int p = 0; p < passes; p++) {
    const int w = total / passes + (p < total % passes ? 1 : 0);
    const uint32_t mask = (1u << w) - 1;
    for (int i = lane; i < kRsSmallPairs; i += 32) my[i] = 0;
    __syncwarp();
    uint32_t rank[kRsItems / 2];
#pragma unroll
    for (int r = 0; r < kRsItems; r++) {
      if (r < rounds) {
        const uint32_t rk = rs_rank<kRsSmallBits>(my16, (uint32_t)(key[r] >> shift) & mask, lt, gt);
        rank[r / 2] = r & 1 ? rank[r / 2] | (rk << 16) : rk;
      }
    }
    __syncthreads();
    {
      const int t = threadIdx.x;
      uint32_t run = 0;
      if (t < kRsSmallPairs) {
#pragma unroll 8
        for (int q = 0; q < kRsSmallWarps; q++) {
          const uint32_t v = cnt[q * kRsSmallPairs + t];
          cnt[q * kRsSmallPairs + t] = run;
          run += v;
        }
      }
      const uint32_t c0 = run & 0xffffu, c1 = run >> 16;
      uint32_t all;
      const uint32_t start = block_excl_scan(c0 + c1, scan_sh, &all);
      if (t < kRsSmallPairs) {
        const uint32_t add = start | ((start + c0) << 16);
#pragma unroll 8
        for (int q = 0; q < kRsSmallWarps; q++) cnt[q * kRsSmallPairs + t] += add;
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kRsItems; r++) {
      if (r < rounds) {
        const uint32_t rk = r & 1 ? rank[r / 2] >> 16 : rank[r / 2] & 0xffffu;
        buf[my16[(uint32_t)(key[r] >> shift) & mask] + rk] = key[r];
      }
    }
    __syncthreads();
    if (p + 1 < passes) {
#pragma unroll
      for (int r = 0; r < kRsItems; r++)
        if (r < rounds) key[r] = buf[i0 + r * 32];
    }
    shift += w;
  }
  // sorted: keep the first of equal keys that FULL and HEAD do not have
  uint32_t kept = 0, found = 0;  // bit r: this lane's key of round r; the warp's count
#pragma unroll
  for (int g = 0; g < kRsItems; g += kDdKeys) {
    if (g < rounds) {
      uint64_t k[kDdKeys];
      bool keep[kDdKeys], hit[kDdKeys];
#pragma unroll
      for (int q = 0; q < kDdKeys; q++) {
        const uint32_t i = i0 + (g + q) * 32;
        const K c = g + q < rounds ? buf[i] : K(0);
        keep[q] = g + q < rounds && i < n && (i == 0 || buf[i - 1] != c);
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
        kept |= (keep[q] ? 1u : 0u) << (g + q);
        found += __popc(__ballot_sync(kAllLanes, keep[q]));
      }
    }
  }
  uint32_t tot;
  // (lane 0 carries the warp's count, so the warp's first position is its prefix)
  uint32_t pos = block_excl_scan(lane == 0 ? found : 0u, scan_sh, &tot);
  pos = __shfl_sync(kAllLanes, pos, 0);
#pragma unroll
  for (int r = 0; r < kRsItems; r++) {
    if (r < rounds) {
      const bool f = (kept >> r) & 1u;
      const unsigned m = __ballot_sync(kAllLanes, f);
      if (f) sel.store(pos + __popc(m & lt), sel.expand(buf[i0 + r * 32]));
      pos += __popc(m);
    }
  }
  if (threadIdx.x == 0) *d_nout = tot;
}

// Lets a scatter kernel use its shared memory on the current device.
template <typename K, int DB, bool FIRST>
static void allow_scatter() {
  static std::atomic<uint64_t> done{0};  // devices the attributes are set on
  int dev = 0;
  SRDL_CUDA(cudaGetDevice(&dev));
  const uint64_t bit = 1ull << (dev & 63);
  if (done.load(std::memory_order_acquire) & bit) return;
  SRDL_CUDA(cudaFuncSetAttribute(rs_scatter<K, DB, FIRST>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 (int)cudaSharedmemCarveoutMaxShared));
  SRDL_CUDA(cudaFuncSetAttribute(rs_scatter<K, DB, FIRST>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)rs_smem_bytes<K, DB>()));
  done.fetch_or(bit, std::memory_order_release);
}

template <typename K>
static void sort_small(const Launch& L, const uint64_t* in, uint64_t n, int bits, bool swap,
                       const DedupDiffSel<K>& sel, uint64_t* d_nout) {
  static std::atomic<uint64_t> done{0};  // devices the attribute is set on
  int dev = 0;
  SRDL_CUDA(cudaGetDevice(&dev));
  const uint64_t bit = 1ull << (dev & 63);
  if (!(done.load(std::memory_order_acquire) & bit)) {
    SRDL_CUDA(cudaFuncSetAttribute(rs_small_kernel<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)rs_small_smem_bytes<K>()));
    done.fetch_or(bit, std::memory_order_release);
  }
  const int passes = (2 * bits + kRsSmallBits - 1) / kRsSmallBits;
  rs_small_kernel<K><<<1, kRsSmallThreads, rs_small_smem_bytes<K>(), L.stream>>>(in, (uint32_t)n, bits, swap, passes,
                                                                                sel, d_nout);
  SRDL_CUDA(cudaGetLastError());
  count_launches(1);
}

// f(std::integral_constant<int, w>) for the digit width w.
template <typename K, typename F>
static void with_digit(int w, F&& f) {
#define SRDL_DIGIT_CASE(DB)                    \
  case DB:                                     \
    f(std::integral_constant<int, DB>{});      \
    return;
  switch (w) {
    SRDL_DIGIT_CASE(1)
    SRDL_DIGIT_CASE(2)
    SRDL_DIGIT_CASE(3)
    SRDL_DIGIT_CASE(4)
    SRDL_DIGIT_CASE(5)
    SRDL_DIGIT_CASE(6)
    SRDL_DIGIT_CASE(7)
    SRDL_DIGIT_CASE(8)
    SRDL_DIGIT_CASE(9)
    default:
      throw Error{kErrState, "radix sort: digit width out of range"};
  }
#undef SRDL_DIGIT_CASE
}

// One counting pass: histogram, offsets, scatter.
template <typename K, bool FIRST>
static void radix_pass(const Launch& L, int nb, int w, const void* in, K* out, uint64_t n, uint64_t chunk, int shift,
                       uint32_t* counts, uint32_t* digit_tot, const uint64_t* d_n, int bits, bool swap) {
  rs_hist<K, FIRST><<<nb, kRsThreads, 0, L.stream>>>(in, n, chunk, shift, 1 << w, counts, d_n, bits, swap);
  rs_rowscan<<<1 << w, kRsScanThreads, 0, L.stream>>>(counts, nb, digit_tot);
  with_digit<K>(w, [&](auto db) {
    constexpr int DB = decltype(db)::value;
    allow_scatter<K, DB, FIRST>();
    rs_scatter<K, DB, FIRST><<<nb, kRsThreads, rs_smem_bytes<K, DB>(), L.stream>>>(
        in, out, n, chunk, shift, counts, digit_tot, d_n, bits, swap);
  });
  SRDL_CUDA(cudaGetLastError());
  count_launches(3);
}

int radix_passes(const Launch& L, int dom_bits) {
  const int maxw = L.radix_bits >= 1 && L.radix_bits <= 7 ? L.radix_bits : kRsAutoBits;
  return (2 * dom_bits + maxw - 1) / maxw;
}

static inline bool use32(int bits) { return 2 * bits <= 32; }

// A bitmap set instead of counting passes (keyset.cu) when the key space is
// small enough and the keys are not too few for it: clearing, counting and
// listing 2^28 bits take about 50 us, a sort of a few ten thousand keys 75-90.
// Measured, set / sort: 3M keys of 2^26 66 / 137 us, 20M of 2^24 174 / 470 us,
// 200k of 2^28 53 / 91 us.  Sorts of one block are beaten from 6,000 keys on where
// the set is at most 2 MB: 9,000 keys of 2^24 39 / 46 us, 5,000 38 / 36.  The
// caller's scratch has to have room for the set: what srdl_sort_unique_u64 states
// has it from about 770,000 keys of 2^26 and 3.9M of 2^28 on, and the runtime's
// own sorts ask for it unless a run's memory is limited.
// FULL and HEAD are read whole to take their keys out of a set, and searched once
// per key otherwise, so they are compared with the keys.  70k keys of 2^26 against
// 10M of FULL 59 / 77 us and against 30M 140 / 81; 1M against 30M 146 / 152 and,
// of 2^28, against 100M 406 / 224; 4M against 100M 426 / 452.
constexpr uint64_t kKeysetSpacePerKey = 4096;
constexpr uint64_t kKeysetMinKeys = 6000;
constexpr uint64_t kKeysetKnown = 12u << 20, kKeysetKnownPerKey = 16;

bool sort_by_keyset(uint64_t n, int bits, uint64_t n_known) {
  return n > (2 * bits <= 24 ? kKeysetMinKeys : kRsSmall) && 2 * bits <= kKeysetMaxBits &&
         n >= (1ull << (2 * bits)) / kKeysetSpacePerKey && n_known <= kKeysetKnown + kKeysetKnownPerKey * n;
}

size_t sort_dev_scratch_bytes(uint64_t cap, uint64_t full_cap, int bits) {
  return sort_scratch_bytes(cap, bits) + diff_dev_extra_bytes(cap, full_cap);
}

size_t sort_scratch_bytes(uint64_t n, int bits) {
  const size_t ks = use32(bits) ? 4 : 8;
  const size_t counts = (size_t)256 * 256 * 8 * 4;  // 2^9 digits of 4 blocks, or 2^10 of 2, on each of 256 SMs
  return 2 * (((n * ks) + 255) & ~size_t(255)) + counts + 2048 + cp_scratch_bytes(n) + 1024;
}

template <typename K>
static void sort_dedup_t(const Launch& L, const uint64_t* in, uint64_t n, int bits, bool swap,
                         const uint64_t* full, uint64_t n_full, uint64_t* out,
                         uint64_t* d_nout, Scratch& s, const uint64_t* head, uint64_t n_head,
                         const uint64_t* d_n, const uint64_t* d_n_full, uint64_t out_cap = ~0ull,
                         unsigned int* d_overflow = nullptr) {
  SRDL_REQUIRE(n < (1ull << 32), kErrCapacity, "sort: more than 2^32-1 rows in one index");
  K* a = s.take<K>(n);
  K* b = s.take<K>(n);
  if (!d_n && n <= kRsSmall) {
    DedupDiffSel<K> sel{nullptr, bits, true, full, full ? n_full : 0, out, head, head ? n_head : 0};
    sort_small<K>(L, in, n, bits, swap, sel, d_nout);
    return;
  }
  // Even split of the keys over the resident blocks, shared by the histogram
  // and scatter launches (with the count on the device, the blocks derive the
  // same split from it).
  const uint64_t resident = (uint64_t)L.num_sms * kRsBlocksPerSm;
  const int nb = (int)std::min<uint64_t>(resident, (n + kRsMinChunk - 1) / kRsMinChunk);
  const uint64_t chunk = rs_chunk(n, nb);
  const int total_bits = 2 * bits;
  const int passes = radix_passes(L, bits);
  uint32_t* counts = s.take<uint32_t>((size_t)nb << ((total_bits + passes - 1) / passes));
  uint32_t* digit_tot = s.take<uint32_t>((size_t)1 << kRsMaxBits);

  int shift = 0;
  for (int p = 0; p < passes; p++) {
    const int w = total_bits / passes + (p < total_bits % passes ? 1 : 0);
    if (p == 0) radix_pass<K, true>(L, nb, w, in, b, n, chunk, shift, counts, digit_tot, d_n, bits, swap);
    else radix_pass<K, false>(L, nb, w, a, b, n, chunk, shift, counts, digit_tot, d_n, bits, swap);
    std::swap(a, b);
    shift += w;
  }
  DedupDiffSel<K> sel{a, bits, true, full, n_full, out, head, n_head};
  sel.d_n_full = d_n_full;
  sel.out_cap = out_cap;
  sel.d_overflow = d_overflow;
  if (d_n) compact_diff_dev(L, sel, n, d_n, d_nout, s);
  else compact_diff(L, sel, n, d_nout, s);
}

// One block and bitmap sets take less scratch than counting passes: a region that
// two copies of the packed keys and the counters of 8-bit passes over 2,048-key
// tiles do not fit in is refused whichever path the keys take.
static void require_room(const Launch& L, uint64_t n, int bits, Scratch s) {
  const size_t ks = use32(bits) ? 4 : 8;
  const int nb = cp_blocks(n, cp_chunk(n, L.num_sms));
  s.take<char>(n * ks);
  s.take<char>(n * ks);
  s.take<uint32_t>((size_t)256 * nb);
  s.take<uint32_t>(256);
  s.take<uint32_t>(cp_words(n));
  s.take<uint32_t>(nb);
}

void sort_dedup(const Launch& L, const uint64_t* in, uint64_t n, int bits, bool swap,
                const uint64_t* full, uint64_t n_full, uint64_t* out, uint64_t* d_nout,
                Scratch& s, const uint64_t* head, uint64_t n_head) {
  if (n == 0) {
    SRDL_CUDA(cudaMemsetAsync(d_nout, 0, sizeof(uint64_t), L.stream));
    return;
  }
  SRDL_REQUIRE(n < (1ull << 32), kErrCapacity, "sort: more than 2^32-1 rows in one index");
  require_room(L, n, bits, s);
  if (sort_by_keyset(n, bits, (full ? n_full : 0) + (head ? n_head : 0)) && s.used + keyset_scratch_bytes(L, bits) <= s.cap) {
    keyset_dedup(L, in, n, bits, swap, full, full ? n_full : 0, head, n_head, out, d_nout, s);
    return;
  }
  if (use32(bits))
    sort_dedup_t<uint32_t>(L, in, n, bits, swap, full, n_full, out, d_nout, s, head, n_head,
                           nullptr, nullptr);
  else sort_dedup_t<uint64_t>(L, in, n, bits, swap, full, n_full, out, d_nout, s, head, n_head,
                              nullptr, nullptr);
}

template <typename K>
static void warm_sort_kernels() {
  for (int w = 1; w <= kRsMaxBits; w++)
    with_digit<K>(w, [](auto db) {
      allow_scatter<K, decltype(db)::value, true>();
      allow_scatter<K, decltype(db)::value, false>();
    });
}

void warm_device_loop_kernels(int bits) {
  if (use32(bits)) warm_sort_kernels<uint32_t>();
  else warm_sort_kernels<uint64_t>();
  warm_merge_kernels();
}

void sort_dedup_dev(const Launch& L, const uint64_t* in, uint64_t cap, const uint64_t* d_n,
                    int bits, const uint64_t* full, uint64_t full_cap, const uint64_t* d_n_full,
                    uint64_t* out, uint64_t out_cap, uint64_t* d_nout, unsigned int* d_overflow,
                    Scratch& s) {
  cap = cap ? cap : 1;
  if (use32(bits))
    sort_dedup_t<uint32_t>(L, in, cap, bits, false, full, full_cap, out, d_nout, s, nullptr, 0, d_n,
                           d_n_full, out_cap, d_overflow);
  else sort_dedup_t<uint64_t>(L, in, cap, bits, false, full, full_cap, out, d_nout, s, nullptr, 0,
                              d_n, d_n_full, out_cap, d_overflow);
}

}  // namespace srdl
