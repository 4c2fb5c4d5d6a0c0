// Findere queries of indexes with singleton groups and rows of at most 32
// chunks: position masks and bit-sliced runs.
//
// Scores::score, findere branch (query_stream.rs:670-689; findere.rs:74-105): a
// colour scores a k-window when all z + 1 s-mers of the window hit it. A warp
// takes a tile's windows w0 .. w0 + nw - 1 and probes the s-mers at positions
// 0 .. nw + z - 1, 128 positions at a time:
//
// * Gather: teams of T lanes (a power of two that holds the row's chunks, one
//   per lane) write each position's match flags, one dense word per chunk,
//   into the warp's table; recovered origins set their bits in it. No hit is
//   handled by itself.
// * Runs: a lane takes one chunk's column over a stretch of positions and
//   keeps, for all of its fields at once, the length of the run of hits in
//   bit-sliced counters that fill at z + 1. A position whose counter is full
//   ends a scoring window; those masks are counted in bit planes. Stretches
//   start z positions early (the table keeps the last z of the 128 before).
//
// The per-hit form (FindereSink, findere_sweep) set a bit per hit with a
// shared-memory atomic and swept every touched colour of each 32 positions:
// 4.6 ms for 1.39e7 s-mers of 128 colours, H 4, b 8 on a B200. It stays for
// indexes with multi-member groups, 1- or 2-bit fields or wider rows.
#pragma once
#include <stdint.h>

#include "window_probe.cuh"

namespace zx {

constexpr uint32_t kFinderePositions = 128;
constexpr uint32_t kFindereChunks = 32;  // widest row
constexpr int kRunPlanes = 8;            // z + 1 up to 225
constexpr size_t kFindereBlockBytes = 110 * 1024;  // two blocks per SM

// Shared memory of a block: DevIndex copy, colour counters, then per warp the
// keys, valid bits, patterns and rows of 32 seeds, and the position table.
struct FindereSmem {
  static __host__ __device__ size_t table_bytes(uint32_t chunks, int z) {
    return ((size_t)(kFinderePositions + (uint32_t)z) * chunks * 4 + 15) / 16 * 16;
  }
  static __host__ __device__ size_t seed_bytes(uint32_t classes, int hashes) {
    return 32 * 4 + 32 * WideSmem::rows_per_seed(classes, hashes) * 4;
  }
  static __host__ __device__ size_t warp_bytes(int k, uint32_t chunks, uint32_t classes, int hashes,
                                               int z) {
    return FusedSmem::key_bytes(3, k) + 64 + seed_bytes(classes, hashes) + table_bytes(chunks, z);
  }
  static __host__ __device__ size_t total(int k, uint32_t colors, uint32_t chunks, uint32_t classes,
                                          int hashes, int z, const QueryLaunch& l) {
    return FusedSmem::ix_bytes + FusedSmem::counter_bytes(colors, l.smem_counters) +
           (size_t)l.warps * warp_bytes(k, chunks, classes, hashes, z);
  }
};

// Same arguments as fused_query_kernel.
template <int MINB>
__global__ void __launch_bounds__(256, MINB)
    findere_query_kernel(const DevIndex* __restrict__ gix, BatchView bv, SeedParams sp,
                         QueryLaunch lc, uint32_t* __restrict__ partial,
                         uint64_t* __restrict__ counts, unsigned long long* __restrict__ total,
                         uint32_t* __restrict__ err) {
  constexpr uint32_t kFull = 0xFFFFFFFFu;
  extern __shared__ __align__(16) uint8_t smem[];
  DevIndex* six = reinterpret_cast<DevIndex*>(smem);
  uint8_t* p = smem + FusedSmem::ix_bytes;
  const uint32_t colors = gix->colors, classes = gix->classes;
  uint32_t* scount = nullptr;
  if (lc.smem_counters) {
    scount = reinterpret_cast<uint32_t*>(p);
    p += FusedSmem::counter_bytes(colors, 1);
  }
  load_index_smem(gix, six);
  if (scount)
    for (uint32_t c = threadIdx.x; c < colors; c += blockDim.x) scount[c] = 0;
  __syncthreads();
  const DevIndex& ix = *six;
  const int H = ix.hashes, Hp = (H + 3) & ~3, b = ix.bits, lb = log2_bits(b);
  const int z = sp.k - sp.klen;
  const uint32_t ones = field_ones(b), hi = ones << (b - 1), fields = 128u >> lb;
  const uint32_t per_seed = classes * (uint32_t)Hp;
  uint32_t chunks = 0;
  for (uint32_t ci = 0; ci < classes; ++ci) chunks += ix.cls[ci].fp_chunks;
  uint32_t lt = 0;
  while ((1u << lt) < chunks) ++lt;
  const uint32_t T = 1u << lt, nteams = 32u >> lt;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t tl = (uint32_t)lane & (T - 1), team = (uint32_t)lane >> lt;
  uint8_t* wbase = p + (size_t)warp * FindereSmem::warp_bytes(sp.k, chunks, classes, H, z);
  uint64_t* keys = reinterpret_cast<uint64_t*>(wbase);
  uint32_t* kvalid = reinterpret_cast<uint32_t*>(wbase + FusedSmem::key_bytes(3, sp.k));
  uint32_t* pattern = kvalid + 16;
  uint32_t* rows = pattern + 32;
  uint32_t* table = rows + 32 * per_seed;  // row: position - first of the 128 + z

  // This lane's chunk: class, columns and field masks (wide_group's layout).
  const uint8_t* col = nullptr;
  uint32_t stride = 0, roff = 0, g0 = 0, valid = 0, cls = 0;
  {
    uint32_t start = 0;
    for (uint32_t ci = 0; ci < classes; ++ci) {
      const DevClass& C = ix.cls[ci];
      if (tl >= start && tl < start + C.fp_chunks) {
        col = C.data + (uint64_t)(tl - start) * 16u;
        stride = C.row_stride;
        roff = ci * (uint32_t)Hp;
        g0 = (tl - start) * fields;
        cls = ci;
        for (uint32_t bit = 0; bit < 32; ++bit)
          if ((bit & (uint32_t)(b - 1)) < 4u && wide_group(g0, bit, b, lb) < C.groups) valid |= 1u << bit;
      }
      start += C.fp_chunks;
    }
  }
  const uint32_t wpb = blockDim.x >> 5;
  uint32_t t_first = bv.tile_lo + blockIdx.x * wpb + warp, t_end = *bv.ntiles;
  uint32_t t_stride = gridDim.x * wpb, seg = 0;
  if (bv.tile_hi && bv.tile_hi < t_end) t_end = bv.tile_hi;
  if (bv.segments) {
    seg = segment_of(bv.seg_blocks, bv.segments, blockIdx.x);
    t_first = bv.seg_tiles[seg] + (blockIdx.x - bv.seg_blocks[seg]) * wpb + warp;
    t_end = bv.seg_tiles[seg + 1];
    t_stride = (bv.seg_blocks[seg + 1] - bv.seg_blocks[seg]) * wpb;
  }
  const Counters cnt{scount, counts + (uint64_t)seg * colors};

  uint32_t planes[kWinPlanes];
#pragma unroll
  for (int k = 0; k < kWinPlanes; ++k) planes[k] = 0;
  uint32_t counted = 0;  // positions in the planes
  auto flush = [&]() {
    uint32_t any = 0;
#pragma unroll
    for (int k = 0; k < kWinPlanes; ++k) any |= planes[k];
    const DevClass& C = ix.cls[cls];
    while (any) {
      const uint32_t bit = __ffs(any) - 1;
      any &= any - 1;
      uint32_t v = 0;
#pragma unroll
      for (int k = 0; k < kWinPlanes; ++k) v |= ((planes[k] >> bit) & 1u) << k;
      cnt.add(__ldg(C.group_color + wide_group(g0, bit, b, lb)), v);
    }
#pragma unroll
    for (int k = 0; k < kWinPlanes; ++k) planes[k] = 0;
    counted = 0;
  };
  // Run counters count up from `from` to 2^bits in z + 1 hits.
  int bits = 0;
  while ((1 << bits) < z + 1) ++bits;
  const uint32_t from = (1u << bits) - (uint32_t)(z + 1);

  unsigned long long seeds = 0;
  for (uint32_t t = t_first; t < t_end; t += t_stride) {
    const Tile tile = bv.tiles[t];
    const uint32_t npos = tile.nw + (uint32_t)z;
    const uint64_t rb = bv.offsets[tile.record];
    if (tile_smers(bv.pv, rb, tile.w0, npos, sp.klen, sp.lk, keys, kvalid, lane)) {
      seeds += tile.nw;
    } else {
      for (uint32_t i0 = 0; i0 < tile.nw; i0 += 32) {
        const uint32_t i = i0 + lane;
        const bool ok = i < tile.nw && bv.pv.valid(rb + tile.w0 + i, (uint32_t)sp.k);
        seeds += __popc(__ballot_sync(kFull, ok));
      }
    }
    for (uint32_t i = lane; i < (uint32_t)z * chunks; i += 32) table[i] = 0;
    for (uint32_t c0 = 0; c0 < npos; c0 += kFinderePositions) {
      const uint32_t m = min(kFinderePositions, npos - c0);
      for (uint32_t r0 = 0; r0 < m; r0 += 32) {
        const uint32_t n = min(32u, m - r0);
        const uint32_t live = kvalid[(c0 + r0) >> 5];
        RecHit rec{nullptr, 0, 0};
        if ((uint32_t)lane < n && ((live >> lane) & 1u)) {
          const uint64_t key = keys[c0 + r0 + lane];
          const uint64_t first = mixsplit(key, ix.seed), step = splitmix64(first);
          pattern[lane] = (uint32_t)fingerprint(key, ix.seed, b) * ones;
          rec = recovery_lookup(ix.rec, recovery_hash(key, ix.seed));
          uint32_t* my = rows + lane * per_seed;
          for (uint32_t ci = 0; ci < classes; ++ci) {
            const DevClass& C = ix.cls[ci];
            const uint32_t part = C.partitions > 1 ? partition_id(key, ix.seed, C.partitions) : 0;
            const uint64_t count = C.slots / C.seg - (uint64_t)H + 1;
            const uint32_t sg = (uint32_t)C.seg;
            const uint32_t row0 = (uint32_t)((uint64_t)part * C.slots + mulhi64(first, count) * C.seg);
            uint64_t h = first;
            for (int i = 0; i < H; ++i, h += step)
              my[ci * Hp + i] = row0 + (uint32_t)i * sg + (((uint32_t)h ^ (uint32_t)(h >> 33)) & (sg - 1));
          }
        }
        __syncwarp();
        uint32_t* out = table + ((uint32_t)z + r0) * chunks;
        if (tl < chunks) {
          for (uint32_t s0 = team; s0 < n; s0 += 2 * nteams) {
            const uint32_t s1 = s0 + nteams;
            const bool va = (live >> s0) & 1u, vb = s1 < n && ((live >> s1) & 1u);
            uint4 aa, ab;
            gather_xor2(col, stride, rows + s0 * per_seed + roff, rows + (vb ? s1 : s0) * per_seed + roff,
                        H, va, vb, aa, ab);
            const uint32_t wa[4] = {aa.x, aa.y, aa.z, aa.w}, wb[4] = {ab.x, ab.y, ab.z, ab.w};
            const uint32_t pa = pattern[s0], pb = pattern[vb ? s1 : s0];
            uint32_t xa = 0, xb = 0;
#pragma unroll
            for (int w = 0; w < 4; ++w) {
              xa |= zero_fields_hi(wa[w] ^ pa, hi) >> (uint32_t)(b - 1 - w);
              xb |= zero_fields_hi(wb[w] ^ pb, hi) >> (uint32_t)(b - 1 - w);
            }
            out[s0 * chunks + tl] = va ? xa & valid : 0u;
            if (s1 < n) out[s1 * chunks + tl] = vb ? xb & valid : 0u;
          }
        }
        __syncwarp();
        for (uint32_t o = 0; o < rec.len; ++o) {
          const ColorLoc loc = bv.color_loc[rec.at(o)];  // (every colour is in a bank)
          uint32_t chunk = loc.group / fields;
          for (uint32_t ci = 0; ci < (loc.cls_member & 0xFFu); ++ci) chunk += ix.cls[ci].fp_chunks;
          const uint32_t idx = loc.group % fields, fpw = 32u >> lb;
          atomicOr(out + lane * chunks + chunk, 1u << ((idx % fpw) * (uint32_t)b + idx / fpw));
        }
        __syncwarp();
      }
      // Runs: stretches of an odd number of positions (no bank conflicts).
      const uint32_t len = ((m + nteams - 1) / nteams) | 1u;
      const uint32_t a = team * len, e = min(m, a + len);
      if (counted + len > 255u) flush();
      counted += len;
      if (tl < chunks && a < e) {
        uint32_t c[kRunPlanes], full = 0;
#pragma unroll
        for (int k = 0; k < kRunPlanes; ++k) c[k] = (from >> k) & 1u ? kFull : 0u;
        const uint32_t* in = table + tl;
        auto step = [&](uint32_t row) {
          const uint32_t hit = in[row * chunks];
          uint32_t up = hit & ~full;
#pragma unroll
          for (int k = 0; k < kRunPlanes; ++k) {
            if (k >= bits) break;
            const uint32_t x = c[k] & up;
            c[k] ^= up;
            up = x;
            c[k] = (from >> k) & 1u ? c[k] | ~hit : c[k] & hit;
          }
          full = (full | up) & hit;
        };
        // Row a + z is position a; the z rows before it warm the counters up.
        for (uint32_t r = a; r < a + (uint32_t)z; ++r) step(r);
        for (uint32_t i = a; i < e; i += 4) {
          uint32_t d[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            d[u] = 0;
            if (i + (uint32_t)u < e) {
              step(i + (uint32_t)u + (uint32_t)z);
              d[u] = full;
            }
          }
          plane_add4(planes, d);
        }
      }
      __syncwarp();
      // The last z positions go to the front for the next 128.
      if (c0 + m < npos)
        for (uint32_t i0 = 0; i0 < (uint32_t)z * chunks; i0 += 32) {
          const uint32_t i = i0 + lane;
          const uint32_t v = i < (uint32_t)z * chunks ? table[i + m * chunks] : 0u;
          __syncwarp();
          if (i < (uint32_t)z * chunks) table[i] = v;
          __syncwarp();
        }
    }
    __syncwarp();
  }
  flush();
  if (lane == 0 && seeds) atomicAdd(total + seg, seeds);
  __syncthreads();
  if (scount)
    for (uint32_t c = threadIdx.x; c < colors; c += blockDim.x)
      partial[(uint64_t)blockIdx.x * colors + c] = scount[c];
}

}  // namespace zx
