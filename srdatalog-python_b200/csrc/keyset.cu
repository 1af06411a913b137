// keyset.cu -- sets of packed keys as bitmaps over the whole key space.
//
// Datalog creates no values, so a binary relation over values < 2^bits has at
// most 2^(2 bits) tuples.  When that space is small -- 2^26 keys are 8 MB of
// bits, which stay in L2 -- the join output of an iteration is sorted,
// deduplicated and freed of known tuples by setting, clearing and listing bits:
// one pass over the raw keys in place of three launches per radix digit, and
// repeats (a dense closure derives a tuple three to three hundred times) cost
// one L2 operation each instead of a place in every pass.
//
// Same results as the sort and set difference of sort.cu: packed order is key
// order, so the listed bits are the sorted distinct keys.
#include <algorithm>

#include "compact.cuh"
#include "kernels.h"

namespace srdl {

constexpr int kKsThreads = 256;
constexpr int kKsWarps = kKsThreads / 32;
constexpr uint32_t kKsTile = kKsThreads * 4;  // words a block lists at a time

size_t keyset_words(int bits) { return (size_t)1 << (2 * bits > 10 ? 2 * bits - 5 : 5); }

static int ks_blocks(const Launch& L, size_t words) {
  return (int)std::min<uint64_t>((words + kKsTile - 1) / kKsTile, (uint64_t)L.num_sms * 8);
}

size_t keyset_scratch_bytes(const Launch& L, int bits) {
  return keyset_words(bits) * 4 + (size_t)ks_blocks(L, keyset_words(bits)) * 4 + 1024;
}

// Sets the bits of n keys (any order, repeats allowed; halves swapped first
// when `swap` is set).  Bound: L2 atomic operations, one per key.
__global__ void __launch_bounds__(kKsThreads) ks_add_kernel(const uint64_t* __restrict__ in, uint64_t n, int bits,
                                                            bool swap, uint32_t* __restrict__ words) {
  const uint64_t step = (uint64_t)gridDim.x * kKsThreads;
  auto place = [&](uint64_t k) -> uint32_t {
    const uint32_t hi = swap ? (uint32_t)k : (uint32_t)(k >> 32), lo = swap ? (uint32_t)(k >> 32) : (uint32_t)k;
    return ((hi << bits) | lo) & ((1u << (2 * bits)) - 1);  // (values past `bits` bits must not leave the set)
  };
  auto add = [&](uint32_t p) { atomicOr(words + (p >> 5), 1u << (p & 31)); };
  uint64_t i = blockIdx.x * (uint64_t)kKsThreads + threadIdx.x;
  for (; i + 3 * step < n; i += 4 * step) {
    uint64_t k[4];
#pragma unroll
    for (int q = 0; q < 4; q++) k[q] = __ldg(in + i + q * step);
#pragma unroll
    for (int q = 0; q < 4; q++) add(place(k[q]));
  }
  for (; i < n; i += step) add(place(__ldg(in + i)));
}

// Clears (SET: sets) the bits of n sorted keys.  Keys of one word follow one
// another: a warp ORs their bits together and takes one operation per word.
template <bool SET>
__global__ void __launch_bounds__(kKsThreads) ks_sorted_kernel(const uint64_t* __restrict__ keys, uint64_t n, int bits,
                                                               uint32_t* __restrict__ words) {
  const int lane = threadIdx.x & 31;
  const uint64_t step = (uint64_t)gridDim.x * kKsThreads;
  for (uint64_t i0 = blockIdx.x * (uint64_t)kKsThreads + (threadIdx.x & ~31u); i0 < n; i0 += step) {
    const uint64_t i = i0 + lane;
    uint32_t w = 0xffffffffu, b = 0;
    if (i < n) {
      const uint64_t k = __ldg(keys + i);
      const uint32_t p = (((uint32_t)(k >> 32) << bits) | (uint32_t)k) & ((1u << (2 * bits)) - 1);
      w = p >> 5;
      b = 1u << (p & 31);
    }
    const uint32_t before = __shfl_up_sync(kAllLanes, w, 1);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t ob = __shfl_down_sync(kAllLanes, b, d), ow = __shfl_down_sync(kAllLanes, w, d);
      if (lane + d < 32 && ow == w) b |= ob;
    }
    if (i < n && (lane == 0 || before != w)) {
      if (SET) atomicOr(words + w, b);
      else atomicAnd(words + w, ~b);
    }
  }
}

// Bits of each block's `chunk` words (those of `words` that `known` does not
// have, when given).
__global__ void __launch_bounds__(kKsThreads) ks_count_kernel(const uint32_t* __restrict__ words,
                                                              const uint32_t* __restrict__ known, uint32_t nwords,
                                                              uint32_t chunk, uint32_t* __restrict__ counts) {
  __shared__ uint32_t sh[kKsWarps + 1];
  const uint32_t begin = blockIdx.x * chunk, end = min(begin + chunk, nwords);
  uint32_t c = 0;
  for (uint32_t q = begin / 4 + threadIdx.x; q < (end + 3) / 4; q += kKsThreads) {
    uint4 v = __ldg(reinterpret_cast<const uint4*>(words) + q);
    if (known) {
      const uint4 k = __ldg(reinterpret_cast<const uint4*>(known) + q);
      v = make_uint4(v.x & ~k.x, v.y & ~k.y, v.z & ~k.z, v.w & ~k.w);
    }
    c += __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
  }
  uint32_t tot;
  block_excl_scan(c, sh, &tot);
  if (threadIdx.x == 0) counts[blockIdx.x] = tot;
}

// Device loop: an iteration's list pass moves the new keys that FULL does not
// have into it and leaves the set of new keys empty for the next iteration.
// Nothing is changed once the iteration has overflowed.
struct KsDelta {
  uint32_t* full = nullptr;            // FULL's words (null: plain listing)
  uint64_t out_cap = 0;                // room for keys
  const uint64_t* d_full_in = nullptr; // FULL's count before, and where it goes
  uint64_t* d_full_out = nullptr;
  unsigned int* d_overflow = nullptr;
};

// Raises the overflow flag when the counts add up to more than cap: launched
// for every relation of an iteration that computes several before any of them
// is changed.
__global__ void __launch_bounds__(kKsThreads) ks_check_kernel(const uint32_t* __restrict__ counts, int nb, uint64_t cap,
                                                              unsigned int* d_overflow) {
  __shared__ uint64_t sh[kKsWarps + 1];
  const uint64_t total = block_prefix(counts, nb, sh);
  if (threadIdx.x == 0 && total > cap) atomicExch(d_overflow, 1u);
}

// Keys of the set bits, in order.  Lane l of a warp holds words 4l .. 4l + 3 of
// the warp's 128.  Where the bits are many the warp goes over the words that
// are not zero, one lane per bit, so the keys leave in coalesced runs; where
// they are few every lane lists its own (2M keys spread over 2^28 bits took 153
// us with the first way alone, 126 us by radix sort).
template <bool DELTA>
__global__ void __launch_bounds__(kKsThreads) ks_list_kernel(uint32_t* words, uint32_t nwords, uint32_t chunk,
                                                             const uint32_t* __restrict__ counts, int bits,
                                                             uint64_t* __restrict__ out, uint64_t* d_nout, KsDelta kd) {
  __shared__ uint64_t sh[kKsWarps + 1];
  __shared__ uint32_t wtot[2][kKsWarps];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned lt = lanemask_lt();
  const uint32_t lo_mask = (uint32_t)((1ull << bits) - 1);
  uint64_t base = block_prefix(counts, blockIdx.x, sh);
  if (DELTA) {
    // (a flag raised by an earlier launch is the same for every block; so is
    // the total)
    const uint64_t total = block_prefix(counts, gridDim.x, sh);
    if (*kd.d_overflow || total > kd.out_cap) {
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        *d_nout = 0;  // (the iteration is redone: what follows sees no delta)
        atomicExch(kd.d_overflow, 1u);
      }
      return;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      *d_nout = total;
      *kd.d_full_out = *kd.d_full_in + total;
    }
  } else if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
    *d_nout = base + counts[blockIdx.x];
  }
  auto key = [&](uint32_t p) { return ((uint64_t)(p >> bits) << 32) | (p & lo_mask); };
  const uint32_t begin = blockIdx.x * chunk, end = min(begin + chunk, nwords);
  int par = 0;
  for (uint32_t tile = begin; tile < end; tile += kKsTile, par ^= 1) {
    const uint32_t w0 = tile + threadIdx.x * 4;
    uint4 x = make_uint4(0, 0, 0, 0);
    if (w0 < end) {
      x = *reinterpret_cast<const uint4*>(words + w0);
      if (DELTA && (x.x | x.y | x.z | x.w)) {
        *reinterpret_cast<uint4*>(words + w0) = make_uint4(0, 0, 0, 0);
        const uint4 k = *reinterpret_cast<const uint4*>(kd.full + w0);
        x = make_uint4(x.x & ~k.x, x.y & ~k.y, x.z & ~k.z, x.w & ~k.w);
        if (x.x | x.y | x.z | x.w)
          *reinterpret_cast<uint4*>(kd.full + w0) = make_uint4(k.x | x.x, k.y | x.y, k.z | x.z, k.w | x.w);
      }
    }
    const uint32_t mine = __popc(x.x) + __popc(x.y) + __popc(x.z) + __popc(x.w);
    const uint32_t inc = warp_incl_scan(mine);
    if (lane == 31) wtot[par][wid] = inc;
    __syncthreads();
    uint64_t pos = base;
#pragma unroll
    for (int w = 0; w < kKsWarps; w++) {
      const uint32_t c = wtot[par][w];
      pos += w < wid ? c : 0;
      base += c;
    }
    unsigned some = __ballot_sync(kAllLanes, mine != 0);
    if (__reduce_max_sync(kAllLanes, mine) + 4 < 3 * (unsigned)__popc(some)) {
      uint64_t at = pos + inc - mine;
      const uint32_t v[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int q = 0; q < 4; q++)
        for (uint32_t m = v[q]; m; m &= m - 1) out[at++] = key((w0 + q) * 32 + __ffs(m) - 1);
      continue;
    }
    while (some) {
      const int l = __ffs(some) - 1;
      some &= some - 1;
      const uint32_t v[4] = {__shfl_sync(kAllLanes, x.x, l), __shfl_sync(kAllLanes, x.y, l),
                             __shfl_sync(kAllLanes, x.z, l), __shfl_sync(kAllLanes, x.w, l)};
      const uint32_t p0 = (tile + (uint32_t)(wid * 32 + l) * 4) * 32 + lane;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        if ((v[q] >> lane) & 1u) out[pos + __popc(v[q] & lt)] = key(p0 + q * 32);
        pos += __popc(v[q]);
      }
    }
  }
}

static int ks_grid(const Launch& L, uint64_t n) {
  return (int)std::max<uint64_t>(1, std::min<uint64_t>((n + kKsThreads - 1) / kKsThreads, (uint64_t)L.num_sms * 8));
}

static uint32_t ks_chunk(uint32_t nwords, int nb) {
  return (uint32_t)(((nwords + nb - 1) / nb + kKsTile - 1) / kKsTile * kKsTile);
}

void keyset_dedup(const Launch& L, const uint64_t* in, uint64_t n, int bits, bool swap, const uint64_t* full,
                  uint64_t n_full, const uint64_t* head, uint64_t n_head, uint64_t* out, uint64_t* d_nout,
                  Scratch& s) {
  const uint32_t nwords = (uint32_t)keyset_words(bits);
  const int nb = ks_blocks(L, nwords);
  const uint32_t chunk = ks_chunk(nwords, nb);
  uint32_t* words = s.take<uint32_t>(nwords);
  uint32_t* counts = s.take<uint32_t>(nb);
  SRDL_CUDA(cudaMemsetAsync(words, 0, (size_t)nwords * 4, L.stream));
  ks_add_kernel<<<ks_grid(L, (n + 3) / 4), kKsThreads, 0, L.stream>>>(in, n, bits, swap, words);
  if (full && n_full)
    ks_sorted_kernel<false><<<ks_grid(L, n_full), kKsThreads, 0, L.stream>>>(full, n_full, bits, words);
  if (head && n_head)
    ks_sorted_kernel<false><<<ks_grid(L, n_head), kKsThreads, 0, L.stream>>>(head, n_head, bits, words);
  ks_count_kernel<<<nb, kKsThreads, 0, L.stream>>>(words, nullptr, nwords, chunk, counts);
  ks_list_kernel<false><<<nb, kKsThreads, 0, L.stream>>>(words, nwords, chunk, counts, bits, out, d_nout, KsDelta{});
  SRDL_CUDA(cudaGetLastError());
  count_launches(3 + (full && n_full ? 1 : 0) + (head && n_head ? 1 : 0));
}

void keyset_from_sorted(const Launch& L, const uint64_t* keys, uint64_t n, int bits, uint32_t* words) {
  SRDL_CUDA(cudaMemsetAsync(words, 0, keyset_words(bits) * 4, L.stream));
  if (!n) return;
  ks_sorted_kernel<true><<<ks_grid(L, n), kKsThreads, 0, L.stream>>>(keys, n, bits, words);
  SRDL_CUDA(cudaGetLastError());
  count_launches(1);
}

void keyset_list(const Launch& L, uint32_t* words, int bits, uint32_t* counts, uint64_t* out, uint64_t* d_nout) {
  const uint32_t nwords = (uint32_t)keyset_words(bits);
  const int nb = ks_blocks(L, nwords);
  const uint32_t chunk = ks_chunk(nwords, nb);
  ks_count_kernel<<<nb, kKsThreads, 0, L.stream>>>(words, nullptr, nwords, chunk, counts);
  ks_list_kernel<false><<<nb, kKsThreads, 0, L.stream>>>(words, nwords, chunk, counts, bits, out, d_nout, KsDelta{});
  SRDL_CUDA(cudaGetLastError());
  count_launches(2);
}

size_t keyset_counts(const Launch& L, int bits) { return (size_t)ks_blocks(L, keyset_words(bits)); }

void keyset_count_dev(const Launch& L, int bits, const uint32_t* words, const uint32_t* full, uint32_t* counts) {
  const uint32_t nwords = (uint32_t)keyset_words(bits);
  const int nb = ks_blocks(L, nwords);
  ks_count_kernel<<<nb, kKsThreads, 0, L.stream>>>(words, full, nwords, ks_chunk(nwords, nb), counts);
  SRDL_CUDA(cudaGetLastError());
  count_launches(1);
}

void keyset_check_dev(const Launch& L, int bits, const uint32_t* counts, uint64_t out_cap, unsigned int* d_overflow) {
  ks_check_kernel<<<1, kKsThreads, 0, L.stream>>>(counts, ks_blocks(L, keyset_words(bits)), out_cap, d_overflow);
  SRDL_CUDA(cudaGetLastError());
  count_launches(1);
}

void keyset_delta_dev(const Launch& L, int bits, uint32_t* words, uint32_t* full, const uint32_t* counts,
                      uint64_t* out, uint64_t out_cap, uint64_t* d_nout, const uint64_t* d_full_in,
                      uint64_t* d_full_out, unsigned int* d_overflow) {
  const uint32_t nwords = (uint32_t)keyset_words(bits);
  const int nb = ks_blocks(L, nwords);
  ks_list_kernel<true><<<nb, kKsThreads, 0, L.stream>>>(words, nwords, ks_chunk(nwords, nb), counts, bits, out, d_nout,
                                                        KsDelta{full, out_cap, d_full_in, d_full_out, d_overflow});
  SRDL_CUDA(cudaGetLastError());
  count_launches(1);
}

}  // namespace srdl
