// Randstrobemer seeds on the GPU (the Linker, src/anchors.rs:182-256, over
// the candidates of scan, src/anchors.rs:265-353).
//
// Per ACGT run the reference links candidates in position order: every
// canonical k-mer (k-mer indexes), or the run's selected minimizer positions
// sorted and deduplicated (minimizer indexes). Each candidate's partner is the
// first candidate strobe_min..strobe_max bases downstream in the same run
// whose strobe hash differs from it in the fewest of its low 8 bits (the
// candidate itself when there is none); the seed is (h >> 1) + (partner >> 1).
//
// On the device this takes two kernels over the planned tiles:
// * strobe_anchor_kernel marks every candidate in a table indexed by base:
//   bit p of `anchors` when a candidate starts at base p, hashes[p] its strobe
//   hash. A minimizer position selected by several windows is written by each
//   of them with the same value, so the table holds every selected position
//   once, in position order: the reference's sort and deduplication.
// * strobe_link_kernel links each tile's own positions (its windows' starts;
//   the record's last tile also the positions past its last window start,
//   which only minimizer windows select): a forward scan of the table that
//   stops at strobe_max, at the record's end and at the first invalid base
//   (a run break), for any strobe_max. Only the low 8 bits of a candidate's
//   hash decide, so a warp stages those of the next 1,024 positions in shared
//   memory and each lane scans its own stretch (five instructions a
//   candidate). A partner without a differing bit ends a lane's search after
//   256 random candidates on average, and the run of valid bases is followed
//   stage by stage, so the time does not grow with strobe_max: 4 Mbases in
//   records of 100,000, whole call on a B200, 4.6 ms for partners up to 2,000
//   and 4.7 ms up to 60,000 (108 ms when every lane searched to the end). A
//   tile's seeds go to its slot of kStrobeSlot keys, in position order.
//
// Both strands of a record are scored on the device: strobe_reverse_kernel
// makes the reverse complements, strobe_best_kernel keeps the larger count.
#pragma once
#include <stdint.h>

#include "query_kernels.cuh"

namespace zx {

// Shared memory of the anchor kernel: the inner hash table (minimizers),
// then per warp the open-closed minimizer scratch.
struct StrobeSmem {
  static __host__ __device__ size_t warp_bytes(int mode, int k) {
    if (mode != 1) return 0;
    const size_t b = 2 * FusedSmem::ocm_entries(k) * sizeof(Rank16) + (kTileWindows + 1) * 4 + 16;
    return (b + 15) / 16 * 16;
  }
  static __host__ __device__ size_t total(int mode, int k, int warps) {
    return (mode == 1 ? 256 * 8 : 0) + (size_t)warps * warp_bytes(mode, k);
  }
};

__device__ __forceinline__ void strobe_mark(const PackedView& pv, const SeedParams& sp, uint64_t p,
                                            int len, uint32_t* __restrict__ anchors,
                                            uint64_t* __restrict__ hashes) {
  uint64_t key = canonical_at(pv, p, len);
  if (sp.spaced) key = spaced_canonical(sp.pattern, key);
  hashes[p] = strobe_hash(key);
  atomicOr(anchors + (p >> 5), 1u << (p & 31));
}

// MODE 0: k-mer candidates (every valid window). MODE 1: minimizer
// candidates (every window's selected position; every valid m-mer when
// k == m). `anchors` is zeroed before the launch.
template <int MODE>
__global__ void strobe_anchor_kernel(BatchView bv, SeedParams sp, uint32_t* __restrict__ anchors,
                                     uint64_t* __restrict__ hashes, int warps_per_block) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint8_t* inner = nullptr;
  uint8_t* wbase = smem;
  if (MODE == 1) {
    inner = smem;
    wbase = smem + 256 * 8 + (size_t)warp * StrobeSmem::warp_bytes(1, sp.k);
    build_inner_table(sp, inner);
    __syncthreads();
  }
  const bool plain = MODE == 0 || sp.k == sp.m;
  const int len = MODE == 0 ? sp.klen : sp.m;
  const uint32_t ntiles = *bv.ntiles;
  const uint32_t warps_total = gridDim.x * warps_per_block;
  for (uint32_t t = blockIdx.x * warps_per_block + warp; t < ntiles; t += warps_total) {
    const Tile tile = bv.tiles[t];
    const uint64_t rb = bv.offsets[tile.record];
    if (plain) {
      for (uint32_t i = lane; i < tile.nw; i += 32) {
        const uint64_t p = rb + tile.w0 + i;
        if (bv.pv.valid(p, (uint32_t)len)) strobe_mark(bv.pv, sp, p, len, anchors, hashes);
      }
      continue;
    }
    Rank16* pre = reinterpret_cast<Rank16*>(wbase);
    Rank16* suf = pre + FusedSmem::ocm_entries(sp.k);
    uint32_t* pos = reinterpret_cast<uint32_t*>(suf + FusedSmem::ocm_entries(sp.k));
    tile_ocm_select(bv.pv, rb, tile.w0, tile.nw, sp, inner, pre, suf, pos, lane);
    // Windows w0 .. w0 + nw - 1 (index 0 is the previous tile's last window).
    for (uint32_t i = 1 + lane; i <= tile.nw; i += 32)
      if (pos[i] != 0xFFFFFFFFu)
        strobe_mark(bv.pv, sp, rb + tile.w0 - 1 + pos[i], len, anchors, hashes);
    __syncwarp();
  }
}

constexpr uint32_t kStrobeStage = 1024;  // positions whose hash bytes a warp holds
constexpr int kLinkThreads = 256;

// Seeds of every tile into slots[t * kStrobeSlot ...], their number in
// slot_count[t]. len: candidate length (k, or m); extra: positions past a
// record's last window start that can hold candidates (w - 1 for open-closed
// minimizers with k > m, else 0; at most kStrobeExtra); dense: every position
// of a run up to its last len bases is a candidate.
__global__ void __launch_bounds__(kLinkThreads)
    strobe_link_kernel(BatchView bv, SeedParams sp, const uint32_t* __restrict__ anchors,
                       const uint64_t* __restrict__ hashes, int len, uint32_t extra, int dense,
                       uint64_t* __restrict__ slots, uint32_t* __restrict__ slot_count) {
  __shared__ uint8_t stage_bytes[kLinkThreads / 32][kStrobeStage];
  const int lane = threadIdx.x & 31;
  uint8_t* stage = stage_bytes[threadIdx.x >> 5];
  const uint32_t ntiles = *bv.ntiles;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  const uint64_t dmin = max(1u, sp.strobe_min), dmax = sp.strobe_max;
  auto is_anchor = [&](uint64_t p) { return (__ldg(anchors + (p >> 5)) >> (p & 31)) & 1u; };
  for (uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < ntiles; t += warps) {
    const Tile tile = bv.tiles[t];
    const uint64_t rb = bv.offsets[tile.record];
    const uint64_t rlen = bv.offsets[tile.record + 1] - rb;
    const uint64_t windows = rlen >= (uint64_t)sp.k ? rlen - sp.k + 1 : 0;
    // Positions of this tile: its windows' starts, and for the record's
    // last tile the candidate positions past them.
    uint64_t end = tile.w0 + tile.nw;
    if (end == windows && extra) end = min(end + extra, rlen >= (uint64_t)len ? rlen - len + 1 : 0);
    const uint64_t starts = rlen - (uint64_t)len + 1;  // (a tile's record has rlen >= len)
    uint64_t* out = slots + (uint64_t)t * kStrobeSlot;
    uint32_t count = 0;
    for (uint64_t q0 = tile.w0; q0 < end; q0 += 32) {
      const uint64_t q = q0 + lane;
      const bool keep = q < end && is_anchor(rb + q);
      uint64_t h = 0, partner = 0;
      // Partners are at most `most` away; the bases from q + len on are valid
      // as far as `reach`, found stage by stage.
      uint64_t reach = 0, most = 0;
      if (keep) {
        h = partner = __ldg(hashes + rb + q);
        most = min(dmax, starts - 1 - q);
      }
      int fewest = 9;
      const uint64_t far = min(q0 + 31 + dmax, starts - 1);  // last position any lane may use
      for (uint64_t c0 = q0 + dmin; c0 <= far; c0 += kStrobeStage) {
        const uint32_t m = (uint32_t)min((uint64_t)kStrobeStage, far - c0 + 1);
        // (A partner without a differing bit ends its lane's search: among
        // random candidates after 256 on average, whatever strobe_max is.)
        if (!__any_sync(0xFFFFFFFFu, keep && fewest && q + most >= c0)) break;
        if (keep && fewest) {
          const uint64_t need = min(most, c0 + m - 1 > q ? c0 + m - 1 - q : 0);
          while (reach < need) {
            const uint32_t bad = bv.pv.inv32(rb + q + len + reach);
            if (bad) {
              most = min(most, reach + __ffs(bad) - 1);
              break;
            }
            reach += 32;
          }
        }
        __syncwarp();
        for (uint32_t i = lane; i < m; i += 32) stage[i] = (uint8_t)__ldg(hashes + rb + c0 + i);
        __syncwarp();
        if (keep && fewest && most >= dmin && q + most >= c0) {
          const uint32_t lo = q + dmin > c0 ? (uint32_t)(q + dmin - c0) : 0u;
          const uint32_t hi = (uint32_t)min((uint64_t)m - 1, q + most - c0);
          const uint32_t mine = (uint32_t)h & 0xFFu;
          uint32_t best = ~0u;  // differing bits << 16 | place in the stage: the first of the fewest
          if (dense) {
#pragma unroll 4
            for (uint32_t i = lo; i <= hi; ++i) best = min(best, (__popc(mine ^ stage[i]) << 16) | i);
          } else {
            for (uint32_t i0 = lo; i0 <= hi; i0 += 32) {
              // Candidates among positions i0 .. i0 + 31 (bits past hi cleared).
              const uint64_t p = rb + c0 + i0;
              const uint64_t two = (uint64_t)__ldg(anchors + (p >> 5)) |
                                   ((uint64_t)((p & 31) ? __ldg(anchors + (p >> 5) + 1) : 0u) << 32);
              uint32_t x = (uint32_t)(two >> (p & 31));
              if (hi - i0 < 31) x &= (2u << (hi - i0)) - 1u;
              for (; x; x &= x - 1) {
                const uint32_t i = i0 + __ffs(x) - 1;
                best = min(best, (__popc(mine ^ stage[i]) << 16) | i);
              }
            }
          }
          if (best != ~0u && (int)(best >> 16) < fewest) {
            fewest = (int)(best >> 16);
            partner = __ldg(hashes + rb + c0 + (best & 0xFFFFu));
          }
        }
      }
      count = warp_append(out, count, keep, (h >> 1) + (partner >> 1), lane);
    }
    if (lane == 0) slot_count[t] = count;
  }
}

// Reverse complement of every record into out, records in place (src/
// anchors.rs:257-263): A, C, G and T of either case become the upper-case
// complement, every other byte stays. A thread takes 16 bases; offsets that
// the tile planner reports are not followed (bases outside every record stay
// unwritten).
__global__ void strobe_reverse_kernel(const uint8_t* __restrict__ bases, uint64_t nbases,
                                      const uint64_t* __restrict__ offsets, uint64_t records,
                                      uint8_t* __restrict__ out) {
  const uint64_t pieces = (nbases + 15) / 16;
  for (uint64_t x = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; x < pieces;
       x += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t i0 = x * 16, i1 = min(nbases, i0 + 16);
    uint64_t lo = 0, hi = records;  // last record that starts at or before i0
    while (hi - lo > 1) {
      const uint64_t mid = (lo + hi) >> 1;
      if (__ldg(offsets + mid) <= i0) lo = mid;
      else hi = mid;
    }
    for (uint64_t i = i0, r = lo; i < i1; ++i) {
      while (r + 1 < records && __ldg(offsets + r + 1) <= i) ++r;
      const uint64_t a = __ldg(offsets + r), b = __ldg(offsets + r + 1);
      if (i < a || i >= b || b > nbases) continue;
      const uint8_t c = bases[i];
      const uint32_t code = encode_base(c);
      out[a + (b - 1 - i)] = code > 3 ? c : (uint8_t)(0x41434754u >> (8 * code));
    }
  }
}

// counts = the larger of the two strands' counts (records x colours); the
// strands' totals must agree.
__global__ void strobe_best_kernel(uint64_t* __restrict__ counts, const uint64_t* __restrict__ other,
                                   uint64_t n, const unsigned long long* __restrict__ totals,
                                   const unsigned long long* __restrict__ other_totals,
                                   uint64_t records, uint32_t* __restrict__ err) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t c = other[i];
    if (c > counts[i]) counts[i] = c;
    if (i < records && totals[i] != other_totals[i]) atomicOr(err, kErrStrands);
  }
}

// sums[c] += the counts of colour c over the records, *total += their totals:
// kSumRecords records per block.
constexpr uint32_t kSumRecords = 32;
__global__ void sum_records_kernel(const uint64_t* __restrict__ counts,
                                   const unsigned long long* __restrict__ totals, uint64_t records,
                                   uint32_t colors, uint64_t* __restrict__ sums,
                                   unsigned long long* __restrict__ total) {
  const uint64_t r0 = (uint64_t)blockIdx.x * kSumRecords, r1 = min(records, r0 + kSumRecords);
  for (uint32_t c = threadIdx.x; c < colors; c += blockDim.x) {
    unsigned long long s = 0;
    for (uint64_t r = r0; r < r1; ++r) s += counts[r * colors + c];
    if (s) atomicAdd(reinterpret_cast<unsigned long long*>(sums + c), s);
  }
  if (threadIdx.x == 0) {
    unsigned long long s = 0;
    for (uint64_t r = r0; r < r1; ++r) s += totals[r];
    if (s) atomicAdd(total, s);
  }
}

}  // namespace zx
