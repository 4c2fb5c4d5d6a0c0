// Window probe: the dense form of the wide-row probe, gathering from shared
// memory (K5 + K6 for batches whose seeds outnumber the cells).
//
// Same arithmetic as wide_probe_kernel (Index::lookup_selected, src/
// power_merge/storage.rs:2761-2925). It rests on a property of PositionHash
// (storage.rs:3452-3481): a key's H cells lie in H consecutive segments (64
// cells each by default) starting at base = mulhi(first hash, segments - H +
// 1), so base grows with the first hash in every class. In a round sorted by
// the first hash, the seeds of a stretch of buckets therefore read one
// contiguous window of rows: the block copies that window (a slice of w
// 16-byte columns of it) into shared memory once, and every row chunk of
// every seed is then a shared-memory read.
//
// * A slice is w = 1..16 adjacent 16-byte chunks of one class's fingerprint
//   plane. A block takes contiguous runs of the sorted seeds of a slice (the
//   round's seeds times the slices, weighted by their widths, are cut by
//   their number: any skew of the keys leaves the blocks level).
// * Window: `segs` segments from the base of the next seed's bucket. All
//   seeds of the buckets whose bases are at most segs - H segments further
//   are inside; their number is read off the bucket table, so no seed is
//   tested.
// * A warp takes 32 seeds: each lane hashes one and leaves its pattern and
//   the byte offsets of its H rows in the window; then teams of w lanes walk
//   the seeds, lane t of a team owning the slice's chunk t, four seeds at a
//   time. The match flags are counted in eight bit planes per lane (a
//   carry-save adder takes four seeds in 6 logic operations plus the carry)
//   and reach the block's counters every 255 seeds.
// * Recovered origins are counted once per seed, when the keys are sorted
//   (block_count_kernel).
//
// Bound by shared-memory bandwidth: 91 % of the data pipe (128 bytes per clock
// and SM) on rows of 512 chunks H8 b4, 93 % on 256 chunks H3 b16, 78 % on 16
// chunks H4 b8, where the ALU is busy for 68 % (the wide probe was bound by
// L2 latency). B200, kernel time, wide probe -> here:
// 31.4e6 seeds of 256 colours H4 b8 3.41 -> 1.40 ms, 2.4e6 of 16,384 colours H8
// b4 12.64 -> 6.15 ms, 9.5e6 of 2,048 colours H3 b16 15.3 -> 4.73 ms. Warps
// take seeds and blocks take work as they get free: in fixed shares the first
// took 1.79 ms and the last 8.9 ms. Two blocks per SM: one loads a window
// while the other gathers.
#pragma once
#include <stdint.h>

#include "wide_probe.cuh"

namespace zx {

constexpr int kWinThreads = 256;
constexpr int kWinPlanes = 8;              // counts up to 255 per field between flushes
constexpr uint32_t kWinItems = 8;          // small work items per block
constexpr uint32_t kWinBlockBytes = 112 << 10;  // shared memory of a block: two blocks per SM

struct WinSlice {
  uint32_t cls;     // class
  uint32_t chunk0;  // first 16-byte chunk of the class's fingerprint plane
  uint32_t nch;     // chunks (at most 1 << lw)
  uint32_t lw;      // log2 of the slice's width in chunks: lanes per seed
  uint32_t weight;  // cost of a seed in this slice, and the sum of the weights before it
  uint32_t before;
};

struct WinPlan {
  const WinSlice* slices = nullptr;
  uint32_t nslices = 0;
  uint32_t weights = 0;    // sum of the slices' weights
  OrderKey order;          // buckets of the sorted keys
  // The window probe runs a round of at least this many keys, the wide probe
  // a smaller one.
  uint64_t min_keys = ~0ull;
};

// Shared memory: the window, per warp 32 seeds' row offsets and patterns, and
// the slice's field counters (32 lanes of at most 32 fields) and the next seed.
struct WinSmem {
  static __host__ __device__ uint32_t rows_per_seed(int hashes) { return (uint32_t)((hashes + 3) & ~3); }
  // Bytes of the window (a multiple of 1 KiB).
  static __host__ __device__ uint32_t tile_bytes(int hashes) {
    return (kWinBlockBytes - kWinThreads * (rows_per_seed(hashes) + 1) * 4 - 32 * 32 * 4 - 32) & ~1023u;
  }
};

__device__ __forceinline__ void cp_async_chunk(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ uint4 ld_shared16(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(addr));
  return v;
}

__device__ __forceinline__ uint32_t maj(uint32_t a, uint32_t b, uint32_t c) {
  return (a & b) | (c & (a | b));
}

// Adds four flags words to the planes: a carry-save adder for the first two
// planes, half adders for the carry.
__device__ __forceinline__ void plane_add4(uint32_t (&planes)[kWinPlanes], const uint32_t (&d)[4]) {
  const uint32_t t = planes[0] ^ d[0] ^ d[1], c0 = maj(planes[0], d[0], d[1]);
  const uint32_t c1 = maj(t, d[2], d[3]);
  planes[0] = t ^ d[2] ^ d[3];
  uint32_t m = maj(planes[1], c0, c1);
  planes[1] ^= c0 ^ c1;
#pragma unroll
  for (int k = 2; k < kWinPlanes; ++k) {
    const uint32_t x = planes[k] & m;
    planes[k] ^= m;
    m = x;
  }
}

// One block's run [pos, stop) of a slice's sorted seeds. HT: the hash count (0:
// any, rows folded four at a time); LW: log2 of the slice's width, so that a
// team's strides are constants. B16: 16-bit fields and no multi-member group;
// the fields that differ are then counted as they are, two to a register (a
// two-way minimum with 1 and an add per word instead of the 5.5 logic
// operations of flags and planes).
template <int HT, int LW, bool B16>
__device__ __forceinline__ void window_slice(const DevIndex* __restrict__ ix, const WinSlice& S,
                                             const OrderKey& order, uint64_t pos, uint64_t stop,
                                             const uint64_t* __restrict__ keys,
                                             const uint32_t* __restrict__ bucket_end,
                                             uint8_t* smem, uint64_t* __restrict__ counts) {
  constexpr uint32_t w = 1u << LW, nteams = 32u >> LW, row_bytes = w * 16u;
  constexpr int kStep = w < 4 ? (int)w : 4;  // seeds of a team at a time
  const int H = HT ? HT : ix->hashes, b = B16 ? 16 : ix->bits, lb = log2_bits(b);
  const uint32_t Hp = WinSmem::rows_per_seed(H), tile_bytes = WinSmem::tile_bytes(H);
  const int warp = threadIdx.x >> 5;
  const uint32_t lane = threadIdx.x & 31u, tl = lane & (w - 1), team = lane >> LW;
  uint32_t* offs = reinterpret_cast<uint32_t*>(smem + tile_bytes) + (uint32_t)warp * 32u * Hp;
  uint32_t* pattern = reinterpret_cast<uint32_t*>(smem + tile_bytes) +
                      (uint32_t)kWinThreads * Hp + (uint32_t)warp * 32u;
  // Field counters of the slice, one per field and lane (no two lanes of a
  // warp share a bank).
  uint32_t* scount = reinterpret_cast<uint32_t*>(smem + tile_bytes) +
                     (uint32_t)kWinThreads * (Hp + 1);
  uint32_t* next = scount + 32 * 32;
  const uint32_t tile = smem_u32(smem), lane_base = tile + tl * 16u;
  const uint64_t seed = ix->seed;
  const uint32_t ones = field_ones(b), hi = ones << (b - 1), lo = ~hi;
  const uint32_t fields = 128u >> lb;  // per chunk
  const DevClass& C = ix->cls[S.cls];
  const uint64_t slots = C.slots;
  const uint32_t seg = (uint32_t)C.seg, stride = C.row_stride;
  const uint32_t parts = C.partitions;
  const uint64_t count = slots / seg - (uint64_t)H + 1;  // bases
  const uint32_t segs = tile_bytes / (seg * row_bytes);
  // Dense flag positions of this lane's chunk (bits f * b + word; see
  // wide_group), those of multi-member groups apart.
  uint32_t valid = 0, multi = 0;
  if (tl < S.nch)
    for (uint32_t bit = 0; bit < 32; ++bit) {
      if ((bit & (uint32_t)(b - 1)) >= 4u) continue;
      const uint32_t g = wide_group((S.chunk0 + tl) * fields, bit, b, lb);
      if (g >= C.groups) continue;
      valid |= 1u << bit;
      if (__ldg(C.group_color + g) & kMultiGroup) multi |= 1u << bit;
    }
  for (uint32_t f = threadIdx.x; f < 32u * fields; f += kWinThreads) scount[f] = 0;
  uint32_t planes[kWinPlanes];
#pragma unroll
  for (int k = 0; k < kWinPlanes; ++k) planes[k] = 0;
  uint32_t differ[4] = {0, 0, 0, 0};  // B16: per word, the seeds that each half differed from
  uint32_t counted = 0;               // seeds in the planes (the warp's bound)
  constexpr uint32_t kCounts = B16 ? 65535u : 255u;
  auto flush = [&]() {
    if constexpr (B16) {
#pragma unroll
      for (uint32_t q = 0; q < 4; ++q) {
#pragma unroll
        for (uint32_t f = 0; f < 2; ++f) {
          const uint32_t same = counted - ((differ[q] >> (16 * f)) & 0xFFFFu);
          if (same && ((valid >> (16 * f + q)) & 1u)) atomicAdd(scount + (2 * q + f) * 32u + lane, same);
        }
        differ[q] = 0;
      }
      counted = 0;
      return;
    }
    uint32_t any = 0;
#pragma unroll
    for (int k = 0; k < kWinPlanes; ++k) any |= planes[k];
    while (any) {
      const uint32_t bit = __ffs(any) - 1;
      any &= any - 1;
      uint32_t v = 0;
#pragma unroll
      for (int k = 0; k < kWinPlanes; ++k) v |= ((planes[k] >> bit) & 1u) << k;
      atomicAdd(scount + wide_group(0, bit, b, lb) * 32u + lane, v);
    }
#pragma unroll
    for (int k = 0; k < kWinPlanes; ++k) planes[k] = 0;
    counted = 0;
  };

  while (pos < stop) {
    // The window of the buckets from the next seed's on.
    const uint64_t key0 = __ldg(keys + pos);
    const int fbits = order.fbits;
    const uint32_t fb = (uint32_t)(mixsplit(key0, seed) >> (64 - fbits));
    const uint32_t prefix = order_partition(key0, order);
    const uint32_t part = prefix & (parts - 1);
    const uint32_t seg0 = (uint32_t)(((uint64_t)fb * count) >> fbits);
    // First bucket with a base past segs - H segments (whole buckets only).
    uint64_t cut = 1ull << fbits;
    const uint64_t past = (uint64_t)seg0 + segs - (uint32_t)H + 1;
    if (past < count) cut = (past << fbits) / count;
    const uint64_t bucket = ((uint64_t)prefix << fbits) + cut;
    const uint64_t end = min(stop, (uint64_t)__ldg(bucket_end + bucket - 1));
    {
      const uint64_t row0 = (uint64_t)part * slots + (uint64_t)seg0 * seg;
      const uint64_t left = slots - (uint64_t)seg0 * seg;
      const uint32_t nrows = left < (uint64_t)segs * seg ? (uint32_t)left : segs * seg;
      const uint8_t* src = C.data + row0 * stride + S.chunk0 * 16u;
      __syncthreads();  // the last window has been read
      if (threadIdx.x == 0) *next = 0;
      for (uint32_t i = threadIdx.x; i < nrows << LW; i += kWinThreads) {
        const uint32_t r = i >> LW, c = i & (w - 1);
        if (c < S.nch) cp_async_chunk(tile + i * 16u, src + (uint64_t)r * stride + c * 16u);
      }
      asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
      __syncthreads();
    }
    // The window's seeds, 32 at a time to whichever warp is free (in fixed
    // shares the warps end far apart and wait at the barrier above).
    const uint32_t nseeds = (uint32_t)(end - pos);
    auto take = [&]() {
      uint32_t g = 0;
      if (lane == 0) g = atomicAdd(next, 32u);
      return __shfl_sync(0xFFFFFFFFu, g, 0);
    };
    uint32_t g = take();
    uint64_t key = g + lane < nseeds ? __ldg(keys + pos + g + lane) : 0;
    while (g < nseeds) {
      const uint32_t n = min(nseeds - g, 32u);
      {
        // (Lanes past the last seed leave the window's first row.)
        const uint64_t first = mixsplit(key, seed), step = splitmix64(first);
        pattern[lane] = (uint32_t)fingerprint(key, seed, b) * ones;
        uint32_t row = ((uint32_t)mulhi64(first, count) - seg0) * seg;
        uint64_t h = first;
        uint32_t* my = offs + lane * Hp;
        const bool live = lane < n;
#pragma unroll
        for (int q = 0; q < (HT ? (HT + 3) / 4 : 1); ++q)
          for (int r = 0; r < (HT ? 1 : (int)Hp / 4); ++r) {
            uint32_t o[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint32_t at = (row + (((uint32_t)h ^ (uint32_t)(h >> 33)) & (seg - 1))) * row_bytes;
              o[j] = live && (HT ? 4 * q + j < HT : 4 * r + j < H) ? at : 0u;
              h += step;
              row += seg;
            }
            *reinterpret_cast<uint4*>(my + 4 * (q + r)) = make_uint4(o[0], o[1], o[2], o[3]);
          }
      }
      g = take();
      key = g + lane < nseeds ? __ldg(keys + pos + g + lane) : 0;
      if (counted + w > kCounts) flush();
      counted += w;
      __syncwarp();
#pragma unroll 1
      for (uint32_t i0 = 0; i0 < w; i0 += kStep) {
        const uint32_t s0 = i0 * nteams + team;
        uint32_t d[4] = {0, 0, 0, 0};
#pragma unroll
        for (int s = 0; s < kStep; ++s) {
          const uint32_t sd = s0 + (uint32_t)s * nteams;
          const uint32_t pat = pattern[sd];
          uint4 acc = make_uint4(pat, pat, pat, pat);
          const uint4* my = reinterpret_cast<const uint4*>(offs + sd * Hp);
#pragma unroll
          for (int q = 0; q < (HT ? (HT + 3) / 4 : 1); ++q) {
            for (int r = 0; r < (HT ? 1 : (int)Hp / 4); ++r) {
              const uint4 o4 = my[q + r];
              const uint32_t o[4] = {o4.x, o4.y, o4.z, o4.w};
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                if (HT ? 4 * q + j >= HT : 4 * r + j >= H) continue;
                const uint4 v = ld_shared16(lane_base + o[j]);
                acc.x ^= v.x; acc.y ^= v.y; acc.z ^= v.z; acc.w ^= v.w;
              }
            }
          }
          const uint32_t x[4] = {acc.x, acc.y, acc.z, acc.w};
          if constexpr (B16) {
            const uint32_t dead = n < 32 && sd >= n ? ~0u : 0u;  // past the last seed: all differ
#pragma unroll
            for (int q = 0; q < 4; ++q) differ[q] += __vminu2(x[q] | dead, 0x00010001u);
            continue;
          }
          uint32_t m = 0;
#pragma unroll
          for (int q = 0; q < 4; ++q) m |= (~(((x[q] & lo) + lo) | x[q]) & hi) >> (uint32_t)(b - 1 - q);
          d[s] = m & valid;
        }
        if constexpr (B16) continue;
        if (n < 32) {
#pragma unroll
          for (int s = 0; s < kStep; ++s)
            if (s0 + (uint32_t)s * nteams >= n) d[s] = 0;
        }
        if (multi) {
          // Multi-member groups: decode the members of each hit.
#pragma unroll
          for (int s = 0; s < kStep; ++s) {
            const uint32_t sd = s0 + (uint32_t)s * nteams;
            for (uint32_t x = d[s] & multi; x; x &= x - 1) {
              const uint32_t grp = wide_group((S.chunk0 + tl) * fields, __ffs(x) - 1, b, lb);
              const uint32_t* mg = C.multi + 3 * (__ldg(C.group_color + grp) & ~kMultiGroup);
              const uint32_t off = __ldg(mg), bits = __ldg(mg + 1), firstm = __ldg(mg + 2);
              const uint8_t* rows = C.data + ((uint64_t)part * slots + (uint64_t)seg0 * seg) * stride;
              uint64_t mx = 0;
              for (int r = 0; r < H; ++r)
                mx ^= row_bits(rows + (uint64_t)(offs[sd * Hp + r] / row_bytes) * stride, off, bits);
              while (mx) {
                const uint32_t mb = __ffsll((long long)mx) - 1;
                mx &= mx - 1;
                atomicAdd(reinterpret_cast<unsigned long long*>(counts + __ldg(C.members + firstm + mb)), 1ull);
              }
            }
            d[s] &= ~multi;
          }
        }
        plane_add4(planes, d);
      }
      __syncwarp();
    }
    pos = end;
  }
  flush();
  __syncthreads();
  for (uint32_t f = threadIdx.x; f < S.nch * fields; f += kWinThreads) {
    const uint32_t c = f / fields, field = f % fields;
    uint32_t v = 0;
#pragma unroll
    for (uint32_t k = 0; k < nteams; ++k) v += scount[field * 32u + k * w + c];
    if (v)
      atomicAdd(reinterpret_cast<unsigned long long*>(
                    counts + __ldg(C.group_color + (S.chunk0 + c) * fields + field)),
                (unsigned long long)v);
  }
  __syncthreads();
}

template <int HT, bool B16>
__global__ void __launch_bounds__(kWinThreads, 2)
    window_probe_kernel(const DevIndex* __restrict__ ix, WinPlan plan,
                        const uint64_t* __restrict__ keys,
                        const unsigned long long* __restrict__ nkeys,
                        const uint32_t* __restrict__ bucket_end,
                        unsigned long long* __restrict__ work, uint64_t* __restrict__ counts,
                        unsigned long long* __restrict__ total) {
  const uint64_t nk = *nkeys;
  if (nk < plan.min_keys) return;
  extern __shared__ __align__(16) uint8_t smem[];
  if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(total, (unsigned long long)nk);
  // Items of the slices x seeds in weight units: half of them in one item per
  // block, the rest in kWinItems small ones per block, each taken by whichever
  // block is free. (In equal shares the two blocks of an SM ran at unequal
  // speeds and the slower one finished alone: 4.4 against 2.9 ms for 4.7e6
  // minimizers of 2,048 colours.)
  const uint64_t units = nk * plan.weights, head = units / 2;
  const uint32_t G = gridDim.x, items = G * (1 + kWinItems);
  __shared__ uint32_t taken;
  for (;;) {
    if (threadIdx.x == 0) taken = (uint32_t)atomicAdd(work, 1ull);
    __syncthreads();
    const uint32_t item = taken;
    __syncthreads();
    if (item >= items) break;
    const uint64_t rest = units - head, t = item - (uint64_t)G;
    const uint64_t u0 = item < G ? head * item / G : head + rest * t / (G * kWinItems);
    const uint64_t u1 = item < G ? head * (item + 1) / G : head + rest * (t + 1) / (G * kWinItems);
    for (uint32_t sl = 0; sl < plan.nslices; ++sl) {
      const WinSlice S = plan.slices[sl];
      const uint64_t s_first = nk * S.before, s_end = s_first + nk * S.weight;
      if (s_end <= u0) continue;
      if (s_first >= u1) break;
      const uint64_t pos = u0 <= s_first ? 0 : (u0 - s_first + S.weight - 1) / S.weight;
      const uint64_t stop = u1 >= s_end ? nk : (u1 - s_first + S.weight - 1) / S.weight;
      if (pos >= stop) continue;
      switch (S.lw) {
        case 4: window_slice<HT, 4, B16>(ix, S, plan.order, pos, stop, keys, bucket_end, smem, counts); break;
        case 3: window_slice<HT, 3, B16>(ix, S, plan.order, pos, stop, keys, bucket_end, smem, counts); break;
        case 2: window_slice<HT, 2, B16>(ix, S, plan.order, pos, stop, keys, bucket_end, smem, counts); break;
        case 1: window_slice<HT, 1, B16>(ix, S, plan.order, pos, stop, keys, bucket_end, smem, counts); break;
        default: window_slice<HT, 0, B16>(ix, S, plan.order, pos, stop, keys, bucket_end, smem, counts); break;
      }
    }
  }
}

}  // namespace zx
