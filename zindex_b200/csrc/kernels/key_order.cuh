// Ordered rounds: the counting sort of a round's keys by bucket (order_bucket).
//
// block_count_kernel counts the buckets - in shared memory up to 2^13 of them,
// else with one L2 atomic per key - and looks up each key's recovered origins
// for the window probe, since it has the key in hand; order_scan_kernel makes
// the buckets' places; two passes of tile_scatter_kernel place the keys, by the
// buckets' upper half of the bits, then by all of them. A pass sorts a tile of
// 8,192 keys in shared memory and writes each bin's keys as one run at a place
// reserved with one atomic; 2^5 to 2^9 bins a pass keep the runs long.
//
// B200, 1.2e8 keys, 2^13 buckets: count with recovered origins 0.86 ms, the
// passes 0.72 ms each. (A scatter through global counters, two atomics and a
// lone 8-byte write per key, took 2.0 ms, its count 1.2 ms and the recovered
// origins apart 2.4 ms; one pass over 2^13 buckets with a block's own runs
// left millions of partly written sectors open and took 4.5 ms; tiles of 4,096
// keys at three blocks per SM 0.80 ms a pass.)
#pragma once
#include <stdint.h>

#include "wide_probe.cuh"

namespace zx {

constexpr int kLocalOrderBits = 13;  // buckets that a block counts in shared memory
constexpr uint32_t kLocalBuckets = 1u << kLocalOrderBits;
constexpr int kOrderThreads = 1024;
constexpr int kOrderUnroll = 4;  // keys of a thread in flight

// A block's run of n keys: whole strides of the block, so that loads stay
// aligned.
__device__ __forceinline__ void order_run(uint64_t n, uint64_t& lo, uint64_t& hi) {
  const uint64_t step = kOrderThreads;
  const uint64_t per = ((n + gridDim.x - 1) / gridDim.x + step - 1) / step * step;
  lo = min(n, per * blockIdx.x);
  hi = min(n, lo + per);
}

constexpr size_t kRecFilterBytes = (1ull << kRecFilterBits) / 8;
constexpr size_t kRecQueueBytes = kOrderThreads / 32 * 64 * 8;

// hist: keys per bucket (zeroed before). In a round of at least min_keys keys
// (~0: none; dynamic shared memory then also holds the warps' queues and the
// recovery filter, if the map has one) also the origins of recovered keys that
// the filters miss, into counts. Keys that pass the filter queue up, so that
// every lane of a warp has one to look up.
__global__ void __launch_bounds__(kOrderThreads)
    block_count_kernel(const DevIndex* __restrict__ gix, const ColorLoc* __restrict__ color_loc,
                       const uint64_t* __restrict__ keys,
                       const unsigned long long* __restrict__ nkeys, OrderKey o, uint64_t min_keys,
                       uint32_t* __restrict__ hist, uint64_t* __restrict__ counts) {
  extern __shared__ __align__(16) uint32_t bins[];
  const uint64_t n = *nkeys;
  uint64_t lo, hi;
  order_run(n, lo, hi);
  if (lo >= hi) return;
  const uint32_t buckets = o.buckets();
  const bool local = buckets <= kLocalBuckets;
  uint32_t* filter = bins + (local ? buckets : 0);
  const DevRecovery rec = gix->rec;
  const bool recover = n >= min_keys;
  const bool filtered = recover && rec.filter;
  if (local)
    for (uint32_t b = threadIdx.x; b < buckets; b += kOrderThreads) bins[b] = 0;
  if (filtered)
    for (uint32_t i = threadIdx.x; i < (uint32_t)(kRecFilterBytes / 16); i += kOrderThreads)
      reinterpret_cast<uint4*>(filter)[i] = __ldg(reinterpret_cast<const uint4*>(rec.filter) + i);
  __syncthreads();
  // Per warp: the keys that passed the filter and are not looked up yet (at
  // most 31, and 32 more).
  const uint32_t lane = threadIdx.x & 31;
  uint64_t* queue = reinterpret_cast<uint64_t*>(filter + (filtered ? kRecFilterBytes / 4 : 0)) +
                    (threadIdx.x >> 5) * 64;
  uint32_t queued = 0;
  for (uint64_t i0 = lo; i0 < hi; i0 += kOrderThreads * kOrderUnroll) {
    uint64_t key[kOrderUnroll];
    bool live[kOrderUnroll];
#pragma unroll
    for (int u = 0; u < kOrderUnroll; ++u) {
      const uint64_t i = i0 + (uint64_t)u * kOrderThreads + threadIdx.x;
      live[u] = i < hi;
      key[u] = live[u] ? __ldg(keys + i) : 0;
    }
#pragma unroll
    for (int u = 0; u < kOrderUnroll; ++u)
      if (live[u]) {
        if (local) atomicAdd(bins + order_bucket(key[u], o), 1u);
        else atomicAdd(hist + order_bucket(key[u], o), 1u);
      }
    if (!recover) continue;
#pragma unroll
    for (int u = 0; u < kOrderUnroll; ++u) {
      const uint32_t f = recovery_hash(key[u], o.seed) & ((1u << kRecFilterBits) - 1);
      const bool open = live[u] && (!filtered || ((filter[f >> 5] >> (f & 31)) & 1u));
      const uint32_t ballot = __ballot_sync(0xFFFFFFFFu, open);
      if (open) queue[queued + __popc(ballot & ((1u << lane) - 1u))] = key[u];
      queued += __popc(ballot);
      __syncwarp();
      if (queued >= 32) {
        queued -= 32;
        recover_key(*gix, color_loc, queue[queued + lane], WideCounters{nullptr, counts});
        __syncwarp();
      }
    }
  }
  if (recover && lane < queued)
    recover_key(*gix, color_loc, queue[lane], WideCounters{nullptr, counts});
  if (!local) return;
  __syncthreads();
  for (uint32_t b = threadIdx.x; b < buckets; b += kOrderThreads)
    if (bins[b]) atomicAdd(hist + b, bins[b]);
}

// next[b] = start[b << shift]: the first places of a pass's bins.
__global__ void order_bins_kernel(const uint32_t* __restrict__ start, uint32_t bins, int shift,
                                  uint32_t* __restrict__ next) {
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < bins) next[b] = start[b << shift];
}

constexpr int kTileThreads = 512;
constexpr int kTilePer = 16;                            // keys of a thread
constexpr uint32_t kTileKeys = kTileThreads * kTilePer;  // 8,192
constexpr uint32_t kTileBins = 1024;

struct TileSmem {
  uint64_t key[kTileKeys];
  uint16_t bin[kTileKeys];
  uint32_t count[kTileBins];  // keys of a bin, then the first place of the bin in the tile
  uint32_t place[kTileBins];  // place of the bin's run in the list, less that first place
  uint32_t part[kTileThreads / 32];
  uint32_t first, last;       // bins of the tile: first .. last
};

// One pass: bin = bucket >> shift, next[] the bins' next places. Keys of a
// tile keep no particular order within a bin. A tile whose bins span more
// than kTileBins (few keys in many bins) places its keys one by one.
__global__ void __launch_bounds__(kTileThreads, 2)
    tile_scatter_kernel(const uint64_t* __restrict__ keys,
                        const unsigned long long* __restrict__ nkeys, OrderKey o, int shift,
                        uint32_t* __restrict__ next, uint64_t* __restrict__ out) {
  extern __shared__ __align__(16) uint8_t smem[];
  TileSmem& S = *reinterpret_cast<TileSmem*>(smem);
  const uint64_t n = *nkeys;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (uint64_t t0 = (uint64_t)blockIdx.x * kTileKeys; t0 < n; t0 += (uint64_t)gridDim.x * kTileKeys) {
    const uint32_t m = n - t0 < kTileKeys ? (uint32_t)(n - t0) : kTileKeys;
    if (tid == 0) {
      S.first = ~0u;
      S.last = 0;
    }
    __syncthreads();
    uint64_t key[kTilePer];
    uint32_t bin[kTilePer], lo = ~0u, hi = 0;
#pragma unroll
    for (int u = 0; u < kTilePer; ++u) {
      const uint32_t i = (uint32_t)u * kTileThreads + tid;
      key[u] = i < m ? __ldg(keys + t0 + i) : 0;
    }
#pragma unroll
    for (int u = 0; u < kTilePer; ++u) {
      bin[u] = order_bucket(key[u], o) >> shift;
      if ((uint32_t)u * kTileThreads + tid < m) {
        lo = min(lo, bin[u]);
        hi = max(hi, bin[u]);
      }
    }
    lo = __reduce_min_sync(0xFFFFFFFFu, lo);
    hi = __reduce_max_sync(0xFFFFFFFFu, hi);
    if (lane == 0 && lo <= hi) {
      atomicMin(&S.first, lo);
      atomicMax(&S.last, hi);
    }
    __syncthreads();
    const uint32_t first = S.first, nb = S.last - first + 1;
    if (nb > kTileBins) {
#pragma unroll
      for (int u = 0; u < kTilePer; ++u)
        if ((uint32_t)u * kTileThreads + tid < m) out[atomicAdd(next + bin[u], 1u)] = key[u];
      __syncthreads();
      continue;
    }
    for (uint32_t b = tid; b < nb; b += kTileThreads) S.count[b] = 0;
    __syncthreads();
    // bin[]: the bin within the tile, then also the key's rank in it (16 bits).
#pragma unroll
    for (int u = 0; u < kTilePer; ++u) {
      bin[u] -= first;
      if ((uint32_t)u * kTileThreads + tid < m) bin[u] |= atomicAdd(S.count + bin[u], 1u) << 16;
    }
    __syncthreads();
    // Exclusive scan of the bins (two per thread) and their runs' places.
    {
      const uint32_t b = 2 * tid;
      const uint32_t c0 = b < nb ? S.count[b] : 0, c1 = b + 1 < nb ? S.count[b + 1] : 0;
      uint32_t incl = c0 + c1;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= (uint32_t)d) incl += v;
      }
      if (lane == 31) S.part[warp] = incl;
      __syncthreads();
      uint32_t before = incl - c0 - c1;
      for (uint32_t i = 0; i < warp; ++i) before += S.part[i];
      if (b < nb) {
        S.count[b] = before;
        if (c0) S.place[b] = atomicAdd(next + first + b, c0) - before;
      }
      if (b + 1 < nb) {
        S.count[b + 1] = before + c0;
        if (c1) S.place[b + 1] = atomicAdd(next + first + b + 1, c1) - (before + c0);
      }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kTilePer; ++u)
      if ((uint32_t)u * kTileThreads + tid < m) {
        const uint32_t at = S.count[bin[u] & 0xFFFFu] + (bin[u] >> 16);
        S.key[at] = key[u];
        S.bin[at] = (uint16_t)bin[u];
      }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kTilePer; ++u) {
      const uint32_t j = (uint32_t)u * kTileThreads + tid;
      if (j < m) out[S.place[S.bin[j]] + j] = S.key[j];
    }
    __syncthreads();
  }
}

}  // namespace zx
