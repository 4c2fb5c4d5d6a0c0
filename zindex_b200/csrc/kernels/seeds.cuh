// Seed extraction on sm_100a: one warp per tile of k-windows of one record.
//
// Input is the batch packed by pack_kernel: packed[w] holds bases 32w..32w+31
// as 2-bit codes, first base in the two most significant bits; invalid[w] has
// bit i set when base 32w+i is not A/C/G/T (either case). Every kernel below
// reproduces the reference extractors bit for bit:
//   canonical k-mers, k <= 32 ......... src/lib.rs:645-681
//   polynomial k-mer hashes, k > 32 ... src/lib.rs:683-731
//   open-closed mod-minimizers ........ utils/ocm-minimizers/src/implementation.rs:89-346
//   modimizers ........................ src/lib.rs:796-806
//   findere s-mers .................... src/lib.rs:632-640, src/findere.rs:178-233
#pragma once
#include <stdint.h>

#include "../zx_hash.h"
#include "types.cuh"

namespace zx {

// Byte -> 2-bit code, 4 for anything that is not A/C/G/T.
__device__ __forceinline__ uint32_t dev_code(uint8_t b) { return encode_base(b); }

// Four bases of a word (first in the low byte) -> their 2-bit codes as one
// byte, first base on top, and a bit per base that is not A/C/G/T. Of the
// upper-case letters bits 1 and 2, XORed with bits 2 and 3, are the code; a
// letter is valid when it is the one its code stands for.
__device__ __forceinline__ uint32_t pack4(uint32_t x, uint32_t& inv) {
  const uint32_t u = x & 0xDFDFDFDFu;
  const uint32_t c = ((u >> 1) ^ (u >> 2)) & 0x03030303u;
  const uint32_t pair = (c | (c >> 4)) & 0x00330033u;
  const uint32_t bad = u ^ __byte_perm(0x54474341u, 0, pair | (pair >> 8));
  // Bit 7 of every byte of `bad` that is not zero, gathered in four bits.
  const uint32_t nz = (((bad & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | bad) & 0x80808080u;
  inv = ((nz >> 7) * 0x10204080u) >> 28;
  return (c * 0x40100401u) >> 24;
}

// K0: ASCII bases -> packed 2-bit words + invalid masks. Word w covers bases
// 32w..32w+31; positions past `n` are marked invalid. Bound by its reads and
// writes (1.375 bytes a base); a byte-by-byte decode took 171 us for 150 MB on
// a B200.
__device__ __forceinline__ void pack_word(const uint8_t* __restrict__ bases, uint64_t n,
                                          uint64_t* __restrict__ packed,
                                          uint32_t* __restrict__ invalid, uint64_t w) {
  const uint64_t base = w * 32;
  uint64_t v = 0;
  uint32_t inv = 0;
  if (base + 32 <= n) {
    const uint8_t* p = bases + base;
    uint32_t x[8];
    if (((uintptr_t)p & 15) == 0) {
      const uint4 a = *reinterpret_cast<const uint4*>(p);
      const uint4 b = *reinterpret_cast<const uint4*>(p + 16);
      x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
      x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
    } else {
      // Any alignment: the aligned words that hold the 32 bytes, shifted.
      const uint32_t* q = reinterpret_cast<const uint32_t*>((uintptr_t)p & ~(uintptr_t)3);
      const uint32_t shift = 8u * ((uint32_t)(uintptr_t)p & 3u);
      uint32_t lo = q[0];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint32_t hi = i < 7 || shift ? q[i + 1] : 0u;
        x[i] = __funnelshift_r(lo, hi, shift);
        lo = hi;
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      uint32_t bad;
      const uint32_t codes = pack4(x[i], bad);
      v |= (uint64_t)codes << (56 - 8 * i);
      inv |= bad << (4 * i);
    }
  } else {
    for (int i = 0; i < 32; ++i) {
      const uint32_t c = base + i < n ? dev_code(bases[base + i]) : 4;
      inv |= (uint32_t)(c > 3) << i;
      v |= (uint64_t)(c & 3) << (62 - 2 * i);
    }
  }
  packed[w] = v;
  invalid[w] = inv;
}

__global__ void pack_kernel(const uint8_t* __restrict__ bases, uint64_t n,
                            uint64_t* __restrict__ packed, uint32_t* __restrict__ invalid,
                            uint64_t words) {
  for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < words;
       w += (uint64_t)gridDim.x * blockDim.x)
    pack_word(bases, n, packed, invalid, w);
}

struct PackedView {
  const uint64_t* packed;
  const uint32_t* invalid;

  // The 32 bases starting at global position p, first base most significant.
  __device__ __forceinline__ uint64_t bits32(uint64_t p) const {
    uint64_t w = p >> 5;
    uint32_t r = (uint32_t)(p & 31);
    uint64_t hi = __ldg(packed + w);
    if (!r) return hi;
    uint64_t lo = __ldg(packed + w + 1);
    return (hi << (2 * r)) | (lo >> (64 - 2 * r));
  }
  // Invalid flags of the 32 bases starting at p (bit i = base p+i).
  __device__ __forceinline__ uint32_t inv32(uint64_t p) const {
    uint64_t w = p >> 5;
    uint32_t r = (uint32_t)(p & 31);
    uint64_t m = (uint64_t)__ldg(invalid + w) | ((uint64_t)__ldg(invalid + w + 1) << 32);
    return (uint32_t)(m >> r);
  }
  // True when bases [p, p+len) are all A/C/G/T.
  __device__ __forceinline__ bool valid(uint64_t p, uint32_t len) const {
    while (len >= 32) {
      if (inv32(p)) return false;
      p += 32;
      len -= 32;
    }
    return len == 0 || (inv32(p) & ((1u << len) - 1)) == 0;
  }
  __device__ __forceinline__ uint32_t code(uint64_t p) const {
    return (uint32_t)(__ldg(packed + (p >> 5)) >> (62 - 2 * (p & 31))) & 3;
  }
  // Forward 2-bit value of the len <= 32 bases at p.
  __device__ __forceinline__ uint64_t fwd(uint64_t p, int len) const {
    uint64_t v = bits32(p);
    return len == 32 ? v : v >> (64 - 2 * len);
  }
  // Bases with code >= 2 (G or T) among the len bases at p.
  __device__ __forceinline__ uint32_t gt_count(uint64_t p, uint32_t len) const {
    uint32_t c = 0;
    while (len >= 32) {
      c += __popcll(bits32(p) & 0xAAAAAAAAAAAAAAAAull);
      p += 32;
      len -= 32;
    }
    if (len) c += __popcll((bits32(p) >> (64 - 2 * len)) & 0xAAAAAAAAAAAAAAAAull);
    return c;
  }
};

// Reverse complement of a len-base forward value (len <= 32).
__device__ __forceinline__ uint64_t revcomp(uint64_t fwd, int len) {
  uint64_t y = __brevll(~fwd);
  y = ((y >> 1) & 0x5555555555555555ull) | ((y & 0x5555555555555555ull) << 1);
  return len == 32 ? y : y >> (64 - 2 * len);
}

__device__ __forceinline__ uint64_t canonical_at(const PackedView& pv, uint64_t p, int len) {
  uint64_t f = pv.fwd(p, len), r = revcomp(f, len);
  return f < r ? f : r;
}

// Whether a modimizer index samples the key of this hash (hash % sampling == 0).
__device__ __forceinline__ bool sampled(const SeedParams& sp, uint64_t hash) {
  const uint64_t x = hash * sp.sampling_inverse;
  const int r = sp.sampling_shift;
  return ((x >> r) | (r ? x << (64 - r) : 0)) <= sp.sampling_most;
}

// Whether the len bases at p are all A/C/G/T (the warp together).
__device__ __forceinline__ bool warp_valid(const PackedView& pv, uint64_t p, uint32_t len, int lane) {
  const uint64_t q = p >> 5;
  const uint32_t off = (uint32_t)(p & 31), end = off + len, words = (end + 31) >> 5;
  bool bad = false;
  for (uint32_t w = lane; w < words; w += 32) {
    uint32_t m = __ldg(pv.invalid + q + w);
    if (w == 0) m &= ~0u << off;
    if (w + 1 == words && (end & 31)) m &= (1u << (end & 31)) - 1u;
    bad |= m != 0;
  }
  return !__any_sync(0xFFFFFFFFu, bad);
}

// Appends the keys selected by `keep` (one per lane, order = lane order) to
// the warp buffer; returns the new count (warp-uniform).
__device__ __forceinline__ uint32_t warp_append(uint64_t* buf, uint32_t count, bool keep,
                                                uint64_t key, int lane) {
  uint32_t ballot = __ballot_sync(0xFFFFFFFFu, keep);
  if (keep) buf[count + __popc(ballot & ((1u << lane) - 1))] = key;
  return count + __popc(ballot);
}

// 32 consecutive windows of at most 32 bases, one per lane, from the two or
// three words that the whole warp shares.
//
// Whether lane l's window p0 + l .. p0 + l + k - 1 is all A/C/G/T, for the
// first n lanes (p0 + n + k - 2 is a base of the batch).
__device__ __forceinline__ bool short_valid(const PackedView& pv, uint64_t p0, uint32_t n, int k,
                                            int lane) {
  const uint64_t q = p0 >> 5;
  const uint32_t off = (uint32_t)(p0 & 31), end = off + n + (uint32_t)k - 2;  // last base
  const uint32_t i0 = __ldg(pv.invalid + q), i1 = end >= 32 ? __ldg(pv.invalid + q + 1) : 0u;
  const uint32_t i2 = end >= 64 ? __ldg(pv.invalid + q + 2) : 0u;
  const uint32_t r = off + (uint32_t)lane;
  const uint32_t inv = r < 32 ? __funnelshift_r(i0, i1, r) : __funnelshift_r(i1, i2, r - 32);
  return (uint32_t)lane < n && (inv & (k == 32 ? ~0u : (1u << k) - 1u)) == 0;
}

// Canonical value of lane l's window (meaningful where it is valid).
__device__ __forceinline__ uint64_t short_canonical(const PackedView& pv, uint64_t p0, uint32_t n,
                                                    int k, int lane) {
  const uint64_t q = p0 >> 5;
  const uint32_t off = (uint32_t)(p0 & 31), end = off + n + (uint32_t)k - 2;
  const uint64_t w0 = __ldg(pv.packed + q), w1 = end >= 32 ? __ldg(pv.packed + q + 1) : 0ull;
  const uint64_t w2 = end >= 64 ? __ldg(pv.packed + q + 2) : 0ull;
  const uint32_t r = off + (uint32_t)lane;
  const uint64_t hi = r < 32 ? w0 : w1, lo = r < 32 ? w1 : w2;
  const bool half = r & 16;  // 2r bits: one 32-bit word and 2 (r & 15) bits
  const uint32_t x0 = half ? (uint32_t)hi : (uint32_t)(hi >> 32);
  const uint32_t x1 = half ? (uint32_t)(lo >> 32) : (uint32_t)hi;
  const uint32_t x2 = half ? (uint32_t)lo : (uint32_t)(lo >> 32);
  const uint32_t sh = 2 * (r & 15);
  const uint64_t v = ((uint64_t)__funnelshift_l(x1, x0, sh) << 32) | __funnelshift_l(x2, x1, sh);
  const uint64_t f = k == 32 ? v : v >> (64 - 2 * k), c = revcomp(f, k);
  return f < c ? f : c;
}

// Canonical k-mers (k <= 32) of the nw <= 512 windows from global base p, whose
// bases are all A/C/G/T, in window order: lane l takes the windows l * per ..
// of per = ceil(nw / 32) and rolls them (a window's value from its
// neighbour's costs a third of cutting it out of the packed words). Window i
// goes to buf[i + pad * (i / per)]; pad 1 spreads the lanes' runs over the
// banks.
__device__ __forceinline__ void tile_kmers_run(const PackedView& pv, uint64_t p, uint32_t nw, int k,
                                               uint64_t* buf, uint32_t pad, int lane) {
  const uint32_t per = (nw + 31) / 32, a = (uint32_t)lane * per;
  if (a >= nw) return;
  const uint32_t n = min(per, nw - a);
  uint64_t* out = buf + a + pad * (uint32_t)lane;
  const uint64_t mask = k == 32 ? ~0ull : (1ull << (2 * k)) - 1;
  uint64_t f = pv.fwd(p + a, k), r = revcomp(f, k);
  // The bases after the first window (at most 15 are used).
  uint64_t next = n > 1 ? pv.bits32(p + a + k) : 0;
  out[0] = f < r ? f : r;
  for (uint32_t j = 1; j < n; ++j) {
    const uint64_t c = next >> 62;
    next <<= 2;
    f = ((f << 2) | c) & mask;
    r = (r >> 2) | ((3 - c) << (2 * k - 2));
    out[j] = f < r ? f : r;
  }
}

// Canonical k-mers (k <= 32) of windows [w0, w0+nw) of the record starting at
// global base `rb`, in window order (modimizers: the sampled ones).
__device__ __forceinline__ uint32_t tile_kmers_short(const PackedView& pv, const SeedParams& sp,
                                                     uint64_t rb, uint32_t w0, uint32_t nw, int k,
                                                     bool modimizer, uint64_t* buf, int lane) {
  const uint64_t p = rb + w0;
  if (!modimizer && nw && warp_valid(pv, p, nw + (uint32_t)k - 1, lane)) {
    tile_kmers_run(pv, p, nw, k, buf, 0, lane);
    return nw;
  }
  uint32_t count = 0;
  for (uint32_t i0 = 0; i0 < nw; i0 += 32) {
    const uint32_t n = min(32u, nw - i0);
    bool keep = short_valid(pv, p + i0, n, k, lane);
    const uint64_t key = short_canonical(pv, p + i0, n, k, lane);
    if (modimizer) keep = keep && sampled(sp, mixsplit(key, sp.seed));
    count = warp_append(buf, count, keep, key, lane);
  }
  return count;
}

// quads[x] and quads[256 + x]: the terms of four bases (first in the top bits
// of x) in the forward and in the reverse polynomial of a long k-mer.
__device__ __forceinline__ void build_long_table(uint64_t* quads) {
  for (uint32_t x = threadIdx.x; x < 256; x += blockDim.x) {
    uint64_t f = 0, r = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      f = f * kLongKmerBase + ((x >> (6 - 2 * j)) & 3) + 1;
      r = r * kLongKmerBase + 4 - ((x >> (2 * j)) & 3);
    }
    quads[x] = f;
    quads[256 + x] = r;
  }
}

// Polynomial hashes (k > 32): each lane rolls over a contiguous run of
// windows, restarting with a direct evaluation after invalid bases. Lane runs
// are staged in `tmp` (nw entries) and concatenated in lane order. quads: the
// table of build_long_table (the evaluation then takes four bases at a time:
// base by base it was two thirds of a 49-mer's cost), or null.
__device__ __forceinline__ uint32_t tile_kmers_long(const PackedView& pv, const SeedParams& sp,
                                                    uint64_t rb, uint32_t w0, uint32_t nw, int k,
                                                    bool modimizer, uint64_t* buf, uint64_t* tmp,
                                                    const uint64_t* quads, int lane) {
  const LongKmerConsts& lk = sp.lk;
  const uint64_t base4 = kLongKmerBase * kLongKmerBase * kLongKmerBase * kLongKmerBase;
  const uint32_t per = (nw + 31) / 32;
  const uint32_t a = min(nw, per * lane), e = min(nw, a + per);
  uint32_t n = 0;
  bool live = false;
  uint64_t f = 0, r = 0;
  for (uint32_t i = a; i < e; ++i) {
    uint64_t p = rb + w0 + i;
    if (live) {
      if (pv.inv32(p + k - 1) & 1) {
        live = false;
        continue;
      }
      uint64_t o = pv.code(p - 1), c = pv.code(p + k - 1);
      f = (f - (o + 1) * lk.power) * kLongKmerBase + (c + 1);
      r = (r - (4 - o)) * lk.inverse + (4 - c) * lk.power;
    } else {
      if (!pv.valid(p, k)) continue;
      live = true;
      f = 0;
      r = 0;
      uint64_t wgt = 1;
      int q = 0;
      if (quads) {
        uint64_t v = 0;
        for (; q + 4 <= k; q += 4) {
          if ((q & 31) == 0) v = pv.bits32(p + q);
          const uint32_t x = (uint32_t)(v >> 56);
          v <<= 8;
          f = f * base4 + quads[x];
          r += quads[256 + x] * wgt;
          wgt *= base4;
        }
      }
      for (; q < k; ++q) {
        uint64_t c = pv.code(p + q);
        f = f * kLongKmerBase + (c + 1);
        r += (4 - c) * wgt;
        wgt *= kLongKmerBase;
      }
    }
    uint64_t key = splitmix64((f < r ? f : r) ^ lk.domain);
    if (!modimizer || sampled(sp, mixsplit(key, sp.seed))) tmp[a + n++] = key;
  }
  uint32_t incl = n;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, d);
    if (lane >= d) incl += v;
  }
  uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
  for (uint32_t j = 0; j < n; ++j) buf[incl - n + j] = tmp[a + j];
  __syncwarp();
  return total;
}

// ---- findere s-mers ----------------------------------------------------------
// The canonical s-mer (s = klen bases) at every position w0 + i, i < npos, of
// the record starting at global base rb, by position: keys[i], and bit i % 32
// of valid[i / 32] set when its s bases are all A/C/G/T (scan_canonical_kmers
// per ACGT run, lib.rs:645-731, as findere scans them, findere.rs:178-233).
// k > 32 uses the polynomial hash, each lane rolling over a contiguous range.
// True when it found every position valid without testing each.
__device__ __forceinline__ bool tile_smers(const PackedView& pv, uint64_t rb, uint32_t w0,
                                           uint32_t npos, int s, const LongKmerConsts& lk,
                                           uint64_t* keys, uint32_t* valid, int lane) {
  if (s <= 32) {
    const uint64_t p = rb + w0;
    if (warp_valid(pv, p, npos + (uint32_t)s - 1, lane)) {
      tile_kmers_run(pv, p, npos, s, keys, 0, lane);
      for (uint32_t w = lane; w < (npos + 31) / 32; w += 32)
        valid[w] = npos - w * 32 >= 32 ? ~0u : (1u << (npos - w * 32)) - 1u;
      __syncwarp();
      return true;
    }
    for (uint32_t i0 = 0; i0 < npos; i0 += 32) {
      const uint32_t n = min(32u, npos - i0);
      const bool ok = short_valid(pv, p + i0, n, s, lane);
      const uint64_t key = short_canonical(pv, p + i0, n, s, lane);
      if (ok) keys[i0 + lane] = key;
      const uint32_t bits = __ballot_sync(0xFFFFFFFFu, ok);
      if (lane == 0) valid[i0 >> 5] = bits;
    }
    __syncwarp();
    return false;
  }
  for (uint32_t w = lane; w < (npos + 31) / 32; w += 32) valid[w] = 0;
  __syncwarp();
  const uint32_t per = (npos + 31) / 32;
  const uint32_t a = min(npos, per * lane), e = min(npos, a + per);
  bool live = false;
  uint64_t f = 0, r = 0;
  for (uint32_t i = a; i < e; ++i) {
    const uint64_t p = rb + w0 + i;
    if (live) {
      if (pv.inv32(p + s - 1) & 1) {
        live = false;
        continue;
      }
      const uint64_t o = pv.code(p - 1), c = pv.code(p + s - 1);
      f = (f - (o + 1) * lk.power) * kLongKmerBase + (c + 1);
      r = (r - (4 - o)) * lk.inverse + (4 - c) * lk.power;
    } else {
      if (!pv.valid(p, s)) continue;
      live = true;
      f = 0;
      r = 0;
      uint64_t wgt = 1;
      for (int q = 0; q < s; ++q) {
        const uint64_t c = pv.code(p + q);
        f = f * kLongKmerBase + (c + 1);
        r += (4 - c) * wgt;
        wgt *= kLongKmerBase;
      }
    }
    keys[i] = splitmix64((f < r ? f : r) ^ lk.domain);
    atomicOr(valid + (i >> 5), 1u << (i & 31));
  }
  __syncwarp();
  return false;
}

// ---- open-closed mod-minimizers -------------------------------------------
struct Rank16 {
  uint64_t hash;
  uint32_t cls;
  uint16_t left, right;  // tile-local anchor indices of the tied extremes
};

__device__ __forceinline__ bool rank_lt(const Rank16& a, const Rank16& b) {
  return a.cls != b.cls ? a.cls < b.cls : a.hash < b.hash;
}
// a lies left of b; equal ranks keep the leftmost and rightmost positions.
__device__ __forceinline__ Rank16 rank_min(const Rank16& a, const Rank16& b) {
  if (rank_lt(a, b)) return a;
  if (rank_lt(b, a)) return b;
  Rank16 r = a;
  r.right = b.right;
  return r;
}

constexpr uint32_t kOcmTile = 256;  // windows per minimizer tile

// Selected minimizer positions of windows w0 - 1 .. w0 + nw - 1 (nw <=
// kOcmTile): pos[i] is window w0 - 1 + i's selected m-mer, as an index j
// into the tile's anchors (record position w0 - 1 + j), or ~0 for an invalid
// window. pre/suf hold at least nw + W entries each; inner is the
// 4^s-entry table of inner hash ranks; pos holds nw + 1 entries. This form
// takes windows of any span; tile_ocm_select_wide the usual ones.
__device__ void tile_ocm_select_any(const PackedView& pv, uint64_t rb, uint32_t w0, uint32_t nw,
                                const SeedParams& sp, const uint8_t* inner, Rank16* pre,
                                Rank16* suf, uint32_t* pos, int lane) {
  const int k = sp.k, t = sp.ocm.t, s = sp.ocm.s, w = sp.ocm.w;
  const uint32_t W = (uint32_t)(k - t + 1);
  // Anchor index j <-> anchor position w0 - 1 + j (record coordinates).
  const uint32_t anchors = nw + W;
  const uint64_t smask = (1ull << (2 * s)) - 1;
  for (uint32_t j = lane; j < anchors; j += 32) {
    Rank16 rk;
    rk.left = rk.right = (uint16_t)j;
    rk.cls = 3;
    rk.hash = ~0ull;
    if (w0 + j >= 1) {
      uint64_t p = rb + w0 + j - 1;
      uint64_t tf = pv.fwd(p, t);
      uint32_t lo = ~0u, h0 = 0, hm = 0, hl = 0;
      for (int q = 0; q <= t - s; ++q) {
        const uint32_t h = inner[(tf >> (2 * (t - s - q))) & smask];
        lo = h < lo ? h : lo;
        if (q == 0) h0 = h;
        if (q == (t - s) / 2) hm = h;
        if (q == t - s) hl = h;
      }
      rk.cls = hm == lo ? 0 : ((h0 == lo || hl == lo) ? 1 : 2);
      uint64_t tr = revcomp(tf, t);
      rk.hash = mixsplit(tf < tr ? tf : tr, sp.seed);
    }
    suf[j] = rk;
  }
  __syncwarp();
  // Block prefix / suffix minima over blocks of W anchors.
  for (uint32_t b0 = lane * W; b0 < anchors; b0 += 32 * W) {
    uint32_t b1 = min(anchors, b0 + W);
    Rank16 acc = suf[b0];
    pre[b0] = acc;
    for (uint32_t j = b0 + 1; j < b1; ++j) {
      acc = rank_min(acc, suf[j]);
      pre[j] = acc;
    }
    for (uint32_t j = b1 - 1; j-- > b0;) suf[j] = rank_min(suf[j], suf[j + 1]);
  }
  __syncwarp();
  // Selected positions of windows w0-1 .. w0+nw-1 (index i <-> window w0-1+i).
  for (uint32_t i = lane; i <= nw; i += 32) {
    uint32_t sel = 0xFFFFFFFFu;
    if (w0 + i >= 1) {
      uint64_t st = rb + w0 + i - 1;
      if (pv.valid(st, k)) {
        Rank16 best = (i % W == 0) ? suf[i] : rank_min(suf[i], pre[i + W - 1]);
        uint32_t anchor = pv.gt_count(st, k) > (uint32_t)k / 2 ? best.right : best.left;
        sel = i + (anchor - i) % (uint32_t)w;  // anchor index offset from window index
      }
    }
    pos[i] = sel;
  }
  __syncwarp();
}

// Rank of an anchor or of a run of them in 12 bytes: class and the hash's top
// 62 bits, then the hash's low 2 bits, and the leftmost and rightmost anchors
// (15 bits each) of that rank.
struct OcmRank {
  uint64_t k;
  uint32_t p;
};

// a lies left of b; equal ranks keep the leftmost and rightmost positions.
__device__ __forceinline__ OcmRank ocm_min(const OcmRank& a, const OcmRank& b) {
  const bool less = b.k < a.k;
  OcmRank r{less ? b.k : a.k, less ? b.p : a.p};
  if (a.k == b.k) {  // (seldom: the same t-mer twice)
    const uint32_t x = a.p >> 30, y = b.p >> 30;
    r.p = y < x ? b.p : (x < y ? a.p : (a.p & ~0x7FFFu) | (b.p & 0x7FFFu));
  }
  return r;
}

// Anchors of a lane in tile_ocm_select_wide.
__device__ __forceinline__ uint32_t ocm_per_lane(uint32_t nw, uint32_t W) {
  return (nw + W + 31) / 32;
}

// The ranks of a lane's anchors skip .. n - 1 (the first at base p) and their
// running minima for t <= 16 and LAST = t - s in 4 .. 8, by rolling: the t-mer
// and its reverse complement, and the inner ranks' sliding minimum from
// minima of 2 and 4 that byte registers hold back (last eight ranks in `old`,
// two and four minima in `two` and `four`). Returns the minimum of all.
template <int LAST>
__device__ __forceinline__ OcmRank ocm_ranks(const PackedView& pv, uint64_t p, uint32_t skip,
                                             uint32_t n, uint32_t a0, const SeedParams& sp,
                                             const uint8_t* inner, uint64_t* sk, uint32_t* sp_,
                                             uint64_t* pk, uint32_t* pp) {
  static_assert(LAST >= 4 && LAST <= 8 && LAST % 2 == 0, "inner positions of an anchor");
  constexpr int kBack = LAST - 3 < 4 ? LAST - 3 : 4;  // the second minimum of four, so far back
  const int t = sp.ocm.t, s = sp.ocm.s;
  const uint32_t tmask = t == 16 ? ~0u : (1u << (2 * t)) - 1u, smask = (1u << (2 * s)) - 1u;
  uint64_t v = pv.bits32(p);  // (an anchor's bases: at most 17 + 15)
  uint32_t f = 0, r = 0, two = 0, four = 0;
  uint64_t old = 0;
  auto base = [&]() {
    const uint32_t c = (uint32_t)(v >> 62);
    v <<= 2;
    f = ((f << 2) | c) & tmask;
    r = (r >> 2) | ((3u - c) << (2 * t - 2));
  };
  for (int i = 0; i < s - 1; ++i) base();
  uint32_t h0 = 0, hm = 0, hl = 0, lo = 0;
  auto slide = [&]() {
    base();
    hl = inner[f & smask];
    const uint32_t m2 = min(hl, (uint32_t)old & 0xFFu);
    const uint32_t m4 = min(m2, (two >> 8) & 0xFFu);
    h0 = (uint32_t)(old >> (8 * (LAST - 1))) & 0xFFu;
    hm = (uint32_t)(old >> (8 * (LAST / 2 - 1))) & 0xFFu;
    lo = min(min(m4, (four >> (8 * (kBack - 1))) & 0xFFu), h0);
    old = (old << 8) | hl;
    two = (two << 8) | m2;
    four = (four << 8) | m4;
  };
#pragma unroll
  for (int i = 0; i < LAST; ++i) slide();
  OcmRank run{~0ull, 0};
  for (uint32_t j = 0; j < n; ++j) {
    OcmRank rk{~0ull, 3u << 30};
    if (j >= skip) {
      slide();
      const uint32_t cls = hm == lo ? 0u : (h0 == lo || hl == lo ? 1u : 2u);
      const uint64_t hash = mixsplit((uint64_t)min(f, r), sp.seed);
      rk.k = ((uint64_t)cls << 62) | (hash >> 2);
      rk.p = (uint32_t)hash << 30;
    }
    rk.p |= (a0 + j) * 0x8001u;
    run = j ? ocm_min(run, rk) : rk;
    sk[j] = rk.k;
    sp_[j] = rk.p;
    pk[j] = run.k;
    pp[j] = run.p;
  }
  return run;
}

// tile_ocm_select for windows of more than per = ocm_per_lane(nw, W) anchors:
// lane l holds the anchors l * per .. and keeps their running minima from the
// left (P) and from the right (S); a window's minimum is the S of its first
// anchor, the minima of the whole lanes between (shuffled) and the P of its
// last anchor. Each lane then selects for the windows that start at its
// anchors, rolling their G and T counts. `scratch` holds 24 bytes for each of
// 32 * (per | 1) anchors. (One lane per block of W anchors, as
// tile_ocm_select_any has it, left most of the warp idle: 3.6 ms for 2^18 tiles
// of 2,048-colour minimizer windows on a B200.)
__device__ void tile_ocm_select_wide(const PackedView& pv, uint64_t rb, uint32_t w0, uint32_t nw,
                                     const SeedParams& sp, const uint8_t* inner, uint8_t* scratch,
                                     uint32_t* pos, int lane) {
  constexpr uint32_t kFull = 0xFFFFFFFFu;
  const int k = sp.k, t = sp.ocm.t, s = sp.ocm.s, w = sp.ocm.w;
  const uint32_t W = (uint32_t)(k - t + 1), anchors = nw + W;
  const uint32_t per = ocm_per_lane(nw, W), pitch = per | 1;  // odd: no bank conflicts
  uint64_t* sk = reinterpret_cast<uint64_t*>(scratch);
  uint64_t* pk = sk + 32 * pitch;
  uint32_t* sp_ = reinterpret_cast<uint32_t*>(pk + 32 * pitch);
  uint32_t* pp = sp_ + 32 * pitch;
  const uint32_t a0 = (uint32_t)lane * per, at = (uint32_t)lane * pitch;
  const uint32_t n = a0 < anchors ? min(per, anchors - a0) : 0;
  // Position w0 - 1 of a record's first tile does not exist.
  const uint32_t skip = w0 + a0 == 0 ? 1u : 0u;
  const uint64_t p = rb + w0 + a0 - 1 + skip;  // first existing anchor of the lane
  const uint32_t smask = (1u << (2 * s)) - 1;
  const int last = t - s;
  OcmRank run{~0ull, 0};
  const bool fast = t <= 16 && last >= 4 && last <= 8;
  if (fast && n > skip) {
    if (last == 8) run = ocm_ranks<8>(pv, p, skip, n, a0, sp, inner, sk + at, sp_ + at, pk + at, pp + at);
    else if (last == 6) run = ocm_ranks<6>(pv, p, skip, n, a0, sp, inner, sk + at, sp_ + at, pk + at, pp + at);
    else run = ocm_ranks<4>(pv, p, skip, n, a0, sp, inner, sk + at, sp_ + at, pk + at, pp + at);
  }
  uint64_t v = 0;
  int have = 0;  // bases left in v
  for (uint32_t j = fast && n > skip ? n : 0; j < n; ++j) {
    OcmRank rk{~0ull, 3u << 30};  // no anchor: above every rank of a window
    if (j >= skip) {
      if (have < t) {
        v = pv.bits32(p + (j - skip));
        have = 32;
      }
      const uint64_t tf = v >> (64 - 2 * t);
      v <<= 2;
      --have;
      uint32_t lo = ~0u, h0 = 0, hm = 0, hl = 0;
      for (int q = 0; q <= last; ++q) {
        const uint32_t h = inner[(uint32_t)(tf >> (2 * (last - q))) & smask];
        lo = min(lo, h);
        if (q == 0) h0 = h;
        if (q == last / 2) hm = h;
        hl = h;
      }
      const uint64_t cls = hm == lo ? 0 : (h0 == lo || hl == lo ? 1 : 2);
      const uint64_t tr = revcomp(tf, t);
      const uint64_t hash = mixsplit(tf < tr ? tf : tr, sp.seed);
      rk.k = (cls << 62) | (hash >> 2);
      rk.p = (uint32_t)hash << 30;
    }
    rk.p |= (a0 + j) * 0x8001u;  // left and right
    run = j ? ocm_min(run, rk) : rk;
    sk[at + j] = rk.k;
    sp_[at + j] = rk.p;
    pk[at + j] = run.k;
    pp[at + j] = run.p;
  }
  if (n) {
    OcmRank r{sk[at + n - 1], sp_[at + n - 1]};
    for (uint32_t j = n - 1; j-- > 0;) {
      r = ocm_min(OcmRank{sk[at + j], sp_[at + j]}, r);
      sk[at + j] = r.k;
      sp_[at + j] = r.p;
    }
  }
  // Minima of the mid and of the mid + 1 lanes after this one.
  const uint32_t mid = (W - 1) / per - 1;
  OcmRank m0{0, 0}, m1{0, 0};
  for (uint32_t d = 1; d <= mid + 1; ++d) {
    const OcmRank o{__shfl_down_sync(kFull, run.k, d), __shfl_down_sync(kFull, run.p, d)};
    m0 = m1;
    m1 = d == 1 ? o : ocm_min(m1, o);
  }
  const bool all = warp_valid(pv, rb + (w0 ? w0 - 1 : 0), nw + (uint32_t)k - (w0 ? 0u : 1u), lane);
  __syncwarp();
  const uint32_t inverse = ((1u << 20) + (uint32_t)w - 1) / (uint32_t)w;  // x / w for x < 2^9
  if (a0 + skip <= nw) {
    uint32_t gt = pv.gt_count(p, k);
    const uint32_t m = min(per, nw + 1 - a0);
    // G or T flags of the bases that leave and enter the windows.
    uint64_t out = m > 1 ? pv.bits32(p) : 0, in = m > 1 ? pv.bits32(p + k) : 0;
    if (skip) pos[0] = 0xFFFFFFFFu;
    for (uint32_t j = skip; j < m; ++j) {
      const uint32_t i = a0 + j;
      uint32_t je = j + W - 1 - (mid + 1) * per, le = (uint32_t)lane + mid + 1;
      OcmRank best{sk[at + j], sp_[at + j]};
      if (je >= per) {
        je -= per;
        ++le;
        best = ocm_min(best, m1);
      } else if (mid) {
        best = ocm_min(best, m0);
      }
      best = ocm_min(best, OcmRank{pk[le * pitch + je], pp[le * pitch + je]});
      const uint32_t anchor = gt > (uint32_t)k / 2 ? best.p & 0x7FFFu : (best.p >> 15) & 0x7FFFu;
      const uint32_t d = anchor - i;
      const bool ok = all || pv.valid(p + (j - skip), k);
      pos[i] = ok ? i + d - ((d * inverse) >> 20) * (uint32_t)w : 0xFFFFFFFFu;
      gt += (uint32_t)(in >> 63) - (uint32_t)(out >> 63);
      in <<= 2;
      out <<= 2;
    }
  }
  __syncwarp();
}

// Selected minimizer positions (see tile_ocm_select_any); pre and suf are one
// buffer.
__device__ __forceinline__ void tile_ocm_select(const PackedView& pv, uint64_t rb, uint32_t w0,
                                                uint32_t nw, const SeedParams& sp,
                                                const uint8_t* inner, Rank16* pre, Rank16* suf,
                                                uint32_t* pos, int lane) {
  const uint32_t W = (uint32_t)(sp.k - sp.ocm.t + 1);
  if (W > ocm_per_lane(nw, W))
    tile_ocm_select_wide(pv, rb, w0, nw, sp, inner, reinterpret_cast<uint8_t*>(pre), pos, lane);
  else
    tile_ocm_select_any(pv, rb, w0, nw, sp, inner, pre, suf, pos, lane);
}

// The positions (as pos[]) that the windows [w0, w0+nw) emit, in window order,
// into the uint32 list at pre; returns their number.
__device__ __forceinline__ uint32_t tile_ocm_list(const PackedView& pv, uint64_t rb, uint32_t w0,
                                                  uint32_t nw, const SeedParams& sp,
                                                  const uint8_t* inner, Rank16* pre, Rank16* suf,
                                                  uint32_t* pos, int lane) {
  tile_ocm_select(pv, rb, w0, nw, sp, inner, pre, suf, pos, lane);
  uint32_t* list = reinterpret_cast<uint32_t*>(pre);
  uint32_t count = 0;
  for (uint32_t i0 = 1; i0 <= nw; i0 += 32) {
    const uint32_t i = i0 + lane;
    const uint32_t at = i <= nw ? pos[i] : 0xFFFFFFFFu;
    const bool keep = at != 0xFFFFFFFFu && at != pos[i - 1];
    const uint32_t ballot = __ballot_sync(0xFFFFFFFFu, keep);
    if (keep) list[count + __popc(ballot & ((1u << lane) - 1u))] = at;
    count += __popc(ballot);
  }
  __syncwarp();
  return count;
}

// Minimizers of windows [w0, w0+nw) (nw <= kOcmTile), buffers as for
// tile_ocm_select. Emits in window order, dropping repeats of the previous
// window's selected position within a run.
__device__ uint32_t tile_ocm(const PackedView& pv, uint64_t rb, uint32_t w0, uint32_t nw,
                             const SeedParams& sp, const uint8_t* inner, Rank16* pre,
                             Rank16* suf, uint32_t* pos, uint64_t* buf, int lane) {
  const uint32_t count = tile_ocm_list(pv, rb, w0, nw, sp, inner, pre, suf, pos, lane);
  const uint32_t* list = reinterpret_cast<const uint32_t*>(pre);
  for (uint32_t i = lane; i < count; i += 32)
    buf[i] = canonical_at(pv, rb + w0 - 1 + list[i], sp.m);
  __syncwarp();
  return count;
}

// Full-m-mer special case (k == m): every canonical m-mer.
__device__ __forceinline__ uint32_t tile_ocm_full(const PackedView& pv, const SeedParams& sp,
                                                  uint64_t rb, uint32_t w0, uint32_t nw,
                                                  uint64_t* buf, int lane) {
  return tile_kmers_short(pv, sp, rb, w0, nw, sp.m, false, buf, lane);
}

}  // namespace zx
