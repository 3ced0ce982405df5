// GPU encoders: ORC RLE v1 and RLE v2 files in CODAG's layouts (include/codag.h,
// codag_compress_rlev1/_rlev2).
//
// CODAG encodes on the GPU with one thread per chunk (rlev1/encoder.h:1728-1847 setup_deflate_orig
// / deflate_orig, rlev2/encoder_trans.h:184-357 block_encode_orig driven by compress_gpu_orig
// :482-564), then scans the stream lengths and moves every stream to its aligned offset.  Here:
//   k_encode         one CTA per chunk, see below; the streams go to slots of the caller's workspace;
//   k_scan_offsets   one CTA turns the stream lengths into the aligned offsets (blk_off);
//   k_gather         one CTA per chunk copies its stream to its offset with the alignment
//                    padding zeroed, and fills col_len.
// Nothing is allocated; a stream that overruns its workspace slot, or a file larger than the
// caller's output capacity, is reported in *d_status.
//
// The host producers' writers (../rle_writers.h) look like state machines over
// the values, but where their items (a run, a group of literals) begin and end depends only on
// where the last one ended and on comparisons of neighbouring values:
//   RLE v1: a run starts at p if its first step is in [-128, 127] and the next step equals it; it
//     goes on while the steps stay equal, for at most 129 values.  What lies between runs is
//     literals, in groups of 127.
//   RLE v2: from p, the first three equal values in a row within 128 values start a fixed run, which
//     goes on for at most 128 values; what lies before them, else 128 values, is a variable group.
// So a CTA's front warps take a tile of 3072 values at a time into shared memory and write their comparisons as
// bit masks, then the length that an item starting at each of the values would have, all in parallel;
// one lane follows the lengths from item to item (searching the masks there instead took 480 cycles
// an item).  Meanwhile
// the back warps measure the items of the tile before, one warp per item, sum the sizes, and write
// the items' bytes.  With one warp per chunk running the state machine, an item cost about 9000 warp
// instructions and a chunk had one warp to wait for.
//
// Many small chunks have a CTA of one warp each (Small).
// RLE v2, 256 MiB of 64-bit values: 3.75 ms with a warp per chunk, 0.90 now (2 CTAs of 16 warps per SM,
// which registers allow; 3 or 4 with fewer registers each: 1.26, 1.40; three, four, six, eight
// front warps instead of five: 0.99, 0.93, 0.93, 0.99).  RLE v1,
// 20 MB of 32-bit values: 1.60 ms, 0.12 now.
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "../../../include/codag.h"
#include "../rlev2_widths.h"
#include "capi_common.cuh"

using namespace codag_dev;

namespace {

constexpr uint64_t kOverflow = ~0ull;

// element j of one chunk of the input zero padded past in_bytes (d_in is element aligned)
template <typename T>
struct PaddedChunk {
  const uint8_t* in;
  uint64_t in_bytes;
  uint64_t base;
  __device__ T operator()(uint64_t j) const {
    const uint64_t o = base + j * sizeof(T);
    if (o + sizeof(T) <= in_bytes) return __ldg(reinterpret_cast<const T*>(in + o));
    T v = 0;
    for (uint32_t k = 0; k < sizeof(T); k++)
      if (o + k < in_bytes) v = static_cast<T>(v | (static_cast<T>(in[o + k]) << (8 * k)));
    return v;
  }
};

// Same integer types as the host producer reads the values with.
template <typename T>
struct Wide;
template <>
struct Wide<uint8_t> { using T = unsigned char; };
template <>
struct Wide<uint16_t> { using T = unsigned short; };
template <>
struct Wide<uint32_t> { using T = unsigned int; };
template <>
struct Wide<uint64_t> { using T = unsigned long long; };

// How a chunk is encoded: TILE values whose items are found at a time, by FRONT warps, and BACK warps that encode them
// meanwhile; FRONT = 0: one warp that does one after the other.
template <uint32_t TILE, uint32_t FRONT, uint32_t BACK, uint32_t CTAS>
struct Shape {
  static constexpr bool kAlone = FRONT == 0;
  static constexpr uint32_t kTile = TILE, kFront = kAlone ? 1 : FRONT, kBack = BACK, kCtas = CTAS;
  static constexpr uint32_t kThreads = 32 * (FRONT + BACK);
  static constexpr uint32_t kAhead = 160;  // values of an item beyond the tile (at most 129)
  static constexpr uint32_t kMaskWords = (TILE + kAhead) / 32;
  static constexpr uint32_t kItems = TILE / 2 + 64;  // a literal between runs of three: two items per four values
};
using BigV1 = Shape<3072, 8, 8, 2>;   // tiles of 2048: 1 to 8% slower; of 4000: one CTA per SM
using BigV2 = Shape<3072, 5, 11, 2>;
using Small = Shape<256, 0, 1, 24>;   // tiles of 128 and 32 CTAs: 10% faster up to 128 values, slower above

// A big CTA is busy 7 us with the smallest chunk, and two fit an SM.  So many small chunks have a CTA of one warp each, which
// takes longer over long ones, the more so for RLE v2, whose items cost more.  Measured, us, big | small, 64-bit values,
// RLE v1: 65536 chunks of 64 values 1420 - 1690 | 290 - 340, 16384 of 256 380 - 520 | 94 - 145, 4096 of 1024
// 114 - 196 | 67 - 115; RLE v2: 2070 - 2470 | 316 - 447, 670 - 700 | 132 - 249, 200 - 240 | 112 - 359.
template <bool V1>
bool small_pays(uint64_t n, uint64_t values) {
  return n > 2 * 148 && values <= 2048 && n >= (V1 ? 1 : 6) * values;
}

// one tile: its values, comparisons and items
template <typename T, class S>
struct EncodeTile {
  static constexpr uint32_t kTile = S::kTile, kAhead = S::kAhead, kMaskWords = S::kMaskWords, kItems = S::kItems;
  T val[kTile + kAhead];
  uint32_t a[kMaskWords];  // RLE v1: a run starts here; RLE v2: the third of three equal values
  uint32_t b[kMaskWords];  // RLE v1: the step to the next value equals the one after; RLE v2: equals the value before
  uint16_t len[kTile];     // values of an item that starts here, and whether it is a run (bit 8)
  uint32_t item[kItems];   // start (12 bits), values (8 bits), run (1 bit)
  uint32_t items;
  uint64_t next;           // first value of the tile after
};

template <typename T, class S, bool V1>
struct EncodeShared {
  static constexpr bool kAlone = S::kAlone;
  static constexpr uint32_t kFront = S::kFront, kBack = S::kBack, kCtas = S::kCtas, kItems = S::kItems, BACK = kBack;
  static constexpr uint32_t kThreads = S::kThreads;
  EncodeTile<T, S> tile[kAlone ? 1 : 2];
  uint32_t off[kItems];           // size of each item
  uint32_t end[V1 ? 1 : kItems];  // RLE v2: where it ends in the tile's bytes
  uint32_t how[V1 ? 1 : kItems];  // RLE v2: see ItemV2::pack
  uint32_t part[BACK];
  uint32_t taken[2][2];           // RLE v2: items measured and written so far, of either tile
  uint32_t hist[V1 ? 1 : BACK][32];
  uint64_t red[V1 ? 1 : BACK][128], list[V1 ? 1 : BACK][32];  // PATCHED_BASE: reduced values, patch list
};

template <uint32_t ID, uint32_t WARPS>
__device__ __forceinline__ void group_barrier() {
  asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(32 * WARPS) : "memory");
}

// bytes of one item, which lies inside its slot
struct Bytes {
  uint8_t* p;
  __device__ __forceinline__ void put(uint32_t at, uint32_t b) const { p[at] = static_cast<uint8_t>(b); }
};

__device__ __forceinline__ uint32_t scan_add(uint32_t v, uint32_t lane) {  // inclusive
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t o = __shfl_up_sync(FULL, v, d);
    if (lane >= static_cast<uint32_t>(d)) v += o;
  }
  return v;
}
__device__ __forceinline__ uint64_t max64(uint64_t v) {
  const uint32_t h = static_cast<uint32_t>(v >> 32), hi = __reduce_max_sync(FULL, h);
  return (static_cast<uint64_t>(hi) << 32) | __reduce_max_sync(FULL, h == hi ? static_cast<uint32_t>(v) : 0u);
}
__device__ __forceinline__ uint64_t min64(uint64_t v) { return ~max64(~v); }

// position past everything that leaves room for sums
constexpr uint32_t kFar = 1u << 30;

// Distance from bit 32 w + lane + skip (skip at most 2) of `mask` (xor `flip`) to the first set bit at or
// after it, if that lies within five words; else kFar.
__device__ __forceinline__ uint32_t distance_to_set(const uint32_t* mask, uint32_t flip, uint32_t w, uint32_t skip,
                                                    uint32_t lane) {
  const uint64_t two = (static_cast<uint64_t>(mask[w + 1] ^ flip) << 32) | (mask[w] ^ flip);
  const uint64_t x = two >> (lane + skip);
  uint32_t far = kFar;
#pragma unroll
  for (uint32_t k = 5; k >= 2; k--) {
    const uint32_t v = mask[w + k] ^ flip;
    if (v) far = 32u * k + __ffs(v) - 1u;
  }
  return x ? static_cast<uint32_t>(__ffsll(static_cast<long long>(x))) - 1u : far - (lane + skip);
}

// step from one value to the next as the writer computes it: in the type's own arithmetic, so never
// negative for 32-bit values, and as an int for narrower ones
template <typename T>
__device__ __forceinline__ int64_t step_of(T a, T b) {
  return static_cast<int64_t>(b - a);
}

// number of significant bits rounded up to a representable width
__device__ __forceinline__ uint32_t width_of(uint64_t v) {
  return v2_closest(64u - static_cast<uint32_t>(__clzll(static_cast<long long>(v))));
}
__device__ __forceinline__ uint32_t varint_len(uint64_t v) {
  return (70u - static_cast<uint32_t>(__clzll(static_cast<long long>(v | 1u)))) / 7u;
}
// byte k of the unsigned LEB128 form of v, whose length is len
__device__ __forceinline__ uint32_t varint_byte(uint64_t v, uint32_t k, uint32_t len) {
  return (static_cast<uint32_t>(v >> (7u * k)) & 0x7fu) | (k + 1u < len ? 0x80u : 0u);
}

// --- RLE v1 items ---------------------------------------------------------------------------------
template <typename T, class S>
struct ItemV1 {
  using Shared = EncodeShared<T, S, true>;
  using Tile = EncodeTile<T, S>;

  static __device__ __forceinline__ uint32_t measure(const T* v, uint32_t n, bool run, Shared&, uint32_t, uint32_t,
                                                     uint32_t lane) {
    if (run) return 2u + varint_len(v[0]);
    uint32_t sum = 0;
#pragma unroll
    for (uint32_t q = 0; q < 4; q++)
      if (32u * q + lane < n) sum += varint_len(v[32u * q + lane]);
    return 1u + __reduce_add_sync(FULL, sum);
  }
  static __device__ __forceinline__ void write(const T* v, uint32_t n, bool run, const Bytes& out, Shared&, uint32_t,
                                               uint32_t, uint32_t lane) {
    uint32_t off = 0;
    if (run) {
      const uint32_t len = varint_len(v[0]);
      if (lane < 2u + len) {
        const uint32_t b = lane == 0 ? n - 3u
                           : lane == 1 ? static_cast<uint32_t>(step_of<T>(v[0], v[1]))
                                       : varint_byte(v[0], lane - 2u, len);
        out.put(off + lane, b);
      }
      return;
    }
    if (lane == 0) out.put(off, 0u - n);
    off++;
#pragma unroll
    for (uint32_t q = 0; q < 4; q++) {
      if (32u * q >= n) break;
      const bool on = 32u * q + lane < n;
      const T x = on ? v[32u * q + lane] : T(0);
      const uint32_t len = on ? varint_len(x) : 0u;
      const uint32_t upto = scan_add(len, lane);
      const uint32_t at = off + (upto - len);
      for (uint32_t k = 0; k < len; k++) out.put(at + k, varint_byte(x, k, len));
      off += __shfl_sync(FULL, upto, 31);
    }
  }
};

// --- RLE v2 items (the choices are those of RleV2Writer, ../rle_writers.h) ------------------------------
template <typename T, class S>
struct ItemV2 {
  using Shared = EncodeShared<T, S, false>;
  using Tile = EncodeTile<T, S>;
  enum : uint32_t { kShortRepeat, kDirect, kDeltaFixed, kDelta, kPatched };
  uint64_t v[4];   // value 32 q + lane
  uint64_t first, second, lmin;
  uint32_t n, size, kind, bits;
  uint32_t pwidth, npatch, gap_width;  // kPatched, whose `bits` is the width of the reduced values

  __device__ __forceinline__ uint32_t pack() const {
    return kind | (bits << 3) | (kind == kPatched ? (pwidth << 10) | (npatch << 17) | (gap_width << 25) : 0u);
  }
  __device__ __forceinline__ void unpack(uint32_t p) {
    kind = p & 7u;
    bits = (p >> 3) & 127u;
    pwidth = (p >> 10) & 127u;
    npatch = (p >> 17) & 255u;
    gap_width = p >> 25;
  }

  // suffix sums of the histogram of the width codes of the values less `sub`: lane c has the number of
  // values of code c and above.  Out of line, as are the packers: the kernel waits for instructions
  // more than for anything else.
  static __device__ __noinline__ uint32_t code_suffix(uint64_t v0, uint64_t v1, uint64_t v2, uint64_t v3, uint64_t sub,
                                                      uint32_t n, uint32_t* hist) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t v[4] = {v0, v1, v2, v3};
    __syncwarp();
    hist[lane] = 0;
    __syncwarp();
#pragma unroll
    for (uint32_t q = 0; q < 4; q++)
      if (32u * q + lane < n) atomicAdd(&hist[v2_code(width_of(v[q] - sub))], 1u);
    __syncwarp();
    const uint32_t c = hist[lane];
    return n - (scan_add(c, lane) - c);
  }
  // smallest width that covers all but the top (100 - p)% of the values
  __device__ __forceinline__ uint32_t percentile(uint32_t suffix, uint32_t p) const {
    p = 100u - p;
    const uint32_t left = p == 0 ? 0u : (n * p - 1u) / 100u + 1u;
    const uint32_t m = __ballot_sync(FULL, suffix > left);
    return m ? v2_width(31u - __clz(m)) : 0u;
  }
  static __device__ __forceinline__ uint32_t aligned_bytes(uint32_t count, uint32_t w) { return (count * w + 7u) / 8u; }
  static __device__ __forceinline__ uint64_t zigzag(uint64_t d) {
    const int64_t s = static_cast<int64_t>(d);
    return static_cast<uint64_t>((s << 1) ^ (s >> 63));
  }

  __device__ __forceinline__ void set_direct(uint32_t suffix) {
    kind = kDirect;
    bits = v2_closest_aligned(percentile(suffix, 100));
    size = 2u + aligned_bytes(n, bits);
  }

  __device__ __forceinline__ void load(const T* val, uint32_t count, uint32_t lane) {
    n = count;
#pragma unroll
    for (uint32_t q = 0; q < 4; q++) v[q] = 32u * q + lane < n ? static_cast<uint64_t>(val[32u * q + lane]) : 0ull;
    first = val[0];
    second = val[n > 1u ? 1 : 0];
  }

  __device__ __forceinline__ void choose(bool is_run, Shared& sh, uint32_t warp, uint32_t lane) {
    bits = 0;
    if (is_run && n < 128u) {  // a fixed run that ended before the limit
      const uint32_t nb = (width_of(first) - 1u) / 8u + 1u;
      kind = n <= 10u ? kShortRepeat : kDeltaFixed;
      size = n <= 10u ? 1u + nb : 3u + varint_len(first);
      return;
    }
    uint32_t* hist = sh.hist[warp];
    const auto suffix = [&](uint64_t sub) { return code_suffix(v[0], v[1], v[2], v[3], sub, n, hist); };
    if (n <= 3u) {
      set_direct(suffix(0));
      return;
    }
    const uint64_t initial = second - first;
    uint64_t lo = first, hi = first, md = 0;
    bool inc = true, dec = true, fix = true;
    uint64_t last = 0;
#pragma unroll
    for (uint32_t q = 0; q < 4; q++) {
      uint64_t prev = shfl_up64(v[q], 1);
      if (lane == 0) prev = last;
      last = shfl64(v[q], 31);
      const uint32_t i = 32u * q + lane;
      if (i > 0 && i < n) {
        const uint64_t d = v[q] - prev;
        lo = v[q] < lo ? v[q] : lo;
        hi = v[q] > hi ? v[q] : hi;
        md = d > md ? d : md;
        inc &= prev <= v[q];
        dec &= prev >= v[q];
        fix &= d == initial;
      }
    }
    lmin = min64(lo);
    const uint64_t lmax = max64(hi);
    // subtracting the minimum is taken for unsafe only for a minimum of 0 and a maximum up to 128
    if (!(lmin > 0 || lmax > 128u)) {
      set_direct(suffix(0));
      return;
    }
    if (__all_sync(FULL, fix)) {
      kind = kDeltaFixed;
      size = 2u + varint_len(first) + varint_len(zigzag(initial));
      return;
    }
    if (initial != 0 && (__all_sync(FULL, inc) || __all_sync(FULL, dec))) {
      kind = kDelta;
      bits = v2_closest_aligned(width_of(max64(md)));
      if (bits == 1u) bits = 2u;
      size = 2u + varint_len(first) + varint_len(zigzag(initial)) + aligned_bytes(n - 2u, bits);
      return;
    }
    const uint32_t plain = suffix(0);
    if (percentile(plain, 100) - percentile(plain, 90) <= 1u) {
      set_direct(plain);
      return;
    }
    const uint32_t reduced = suffix(lmin);
    uint32_t b95 = percentile(reduced, 95);
    const uint32_t r100 = percentile(reduced, 100);
    if (r100 == b95) {
      set_direct(plain);
      return;
    }
    // PATCHED_BASE: values above b95 bits keep their low bits and give an entry (gap, high bits) of the
    // patch list, gaps counted from the patch before (0 before the first)
    kind = kPatched;
    pwidth = v2_closest(r100 - b95);
    if (pwidth == 64u) {
      pwidth = 56u;
      b95 = 8u;
    }
    bits = b95;
    const uint64_t mask = (1ull << b95) - 1ull;
    uint32_t max_gap = 0;
    npatch = 0;
    int32_t prev_pos = -1;
#pragma unroll
    for (uint32_t q = 0; q < 4; q++) {
      const uint32_t bq = __ballot_sync(FULL, 32u * q + lane < n && v[q] - lmin > mask);
      for (uint32_t m = bq; m; m &= m - 1u) {
        const int32_t pos = static_cast<int32_t>(32u * q + __ffs(m) - 1u);
        const uint32_t gap = static_cast<uint32_t>(pos - (prev_pos >= 0 ? prev_pos : 0));
        max_gap = max_gap > gap ? max_gap : gap;
        prev_pos = pos;
      }
      npatch += __popc(bq);
    }
    gap_width = max_gap == 0 && npatch != 0 ? 1u : width_of(max_gap);
    size = 4u + base_bytes() + aligned_bytes(n, bits) + aligned_bytes(npatch, v2_closest(gap_width + pwidth));
  }

  // reduced values and patch list of a PATCHED_BASE group, into shared memory
  __device__ __forceinline__ void stage_patched(Shared& sh, uint32_t warp, uint32_t lane) {
    uint64_t lo = first;
#pragma unroll
    for (uint32_t q = 0; q < 4; q++)
      if (32u * q + lane < n) lo = v[q] < lo ? v[q] : lo;
    lmin = min64(lo);
    const uint64_t mask = (1ull << bits) - 1ull;
    uint32_t before = 0;
    int32_t prev_pos = -1;
    __syncwarp();
#pragma unroll
    for (uint32_t q = 0; q < 4; q++) {
      const uint32_t i = 32u * q + lane;
      const uint64_t r = i < n ? v[q] - lmin : 0ull;
      if (i < n) sh.red[warp][i] = r & mask;
      const bool hit = r > mask;
      const uint32_t bq = __ballot_sync(FULL, hit);
      if (hit) {
        const uint32_t below = bq & lanemask_lt(lane);
        const uint32_t prev = below ? 32u * q + 31u - __clz(below) : (prev_pos >= 0 ? static_cast<uint32_t>(prev_pos) : 0u);
        sh.list[warp][before + __popc(below)] = (static_cast<uint64_t>(i - prev) << pwidth) | (r >> bits);
      }
      if (bq) prev_pos = static_cast<int32_t>(32u * q + 31u - __clz(bq));
      before += __popc(bq);
    }
    __syncwarp();
  }
  __device__ __forceinline__ uint32_t base_bytes() const { return width_of(lmin) / 8u + 1u; }

  // x0..x3 are elements lane, 32 + lane, ...; at an aligned width, most significant bit first
  static __device__ __noinline__ void put_aligned(uint8_t* out, uint64_t x0, uint64_t x1, uint64_t x2, uint64_t x3,
                                                  uint32_t count, uint32_t w) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t x[4] = {x0, x1, x2, x3};
    if (w >= 8u) {
      const uint32_t nb = w / 8u;
#pragma unroll
      for (uint32_t q = 0; q < 4; q++) {
        const uint32_t i = 32u * q + lane;
        if (i < count) {
          uint8_t* p = out + i * nb + nb;
          uint64_t y = x[q];
          for (uint32_t j = 0; j < nb; j++, y >>= 8) *--p = static_cast<uint8_t>(y);
        }
      }
      return;
    }
    const uint32_t per = 8u / w;  // 2, 4 or 8 lanes share a byte
#pragma unroll
    for (uint32_t q = 0; q < 4; q++) {
      const uint32_t i = 32u * q + lane;
      uint32_t b = i < count ? (static_cast<uint32_t>(x[q]) & ((1u << w) - 1u)) << (8u - (i % per + 1u) * w) : 0u;
      for (uint32_t d = 1; d < per; d <<= 1) b |= __shfl_xor_sync(FULL, b, d);
      if (i < count && i % per == 0) out[i / per] = static_cast<uint8_t>(b);
    }
  }
  // `count` values of w bits from shared memory, most significant bit first
  static __device__ __noinline__ void put_packed(uint8_t* out, const uint64_t* x, uint32_t count, uint32_t w) {
    const uint32_t tb = count * w;
    for (uint32_t s = 8u * (threadIdx.x & 31u); s < tb; s += 256u) {
      const uint32_t e = s + 8u < tb ? s + 8u : tb;
      uint32_t byte = 0;
      for (uint32_t i = s / w; i * w < e; i++) {
        const uint32_t vs = i * w, ve = vs + w, a = vs > s ? vs : s, b = ve < e ? ve : e;
        byte |= (static_cast<uint32_t>(x[i] >> (ve - b)) & ((1u << (b - a)) - 1u)) << (s + 8u - b);
      }
      out[s / 8u] = static_cast<uint8_t>(byte);
    }
  }

  __device__ __forceinline__ void put_item(const Bytes& out, uint32_t off, Shared& sh, uint32_t warp, uint32_t lane) {
    const uint32_t len = n - 1u;
    if (kind == kShortRepeat) {
      const uint32_t nb = (width_of(first) - 1u) / 8u + 1u;
      if (lane == 0) out.put(off, ((nb - 1u) << 3) | (n - 3u));
      else if (lane <= nb) out.put(off + lane, static_cast<uint32_t>(first >> (8u * (nb - lane))));
      return;
    }
    const uint32_t top = kind == kDirect ? 0x40u : kind == kPatched ? 0x80u : 0xC0u;
    const uint32_t code = kind == kDeltaFixed ? 0u : v2_code(bits);
    if (lane == 0) out.put(off, top | (code << 1) | ((len >> 8) & 1u));
    if (lane == 1) out.put(off + 1, len);
    off += 2;
    if (kind == kDirect) {
      put_aligned(out.p + off, v[0], v[1], v[2], v[3], n, bits);
      return;
    }
    if (kind == kPatched) {
      stage_patched(sh, warp, lane);
      const uint32_t nb = base_bytes(), w2 = v2_closest(gap_width + pwidth);
      if (lane == 0) out.put(off, ((nb - 1u) << 5) | v2_code(pwidth));
      if (lane == 1) out.put(off + 1, ((gap_width - 1u) << 5) | npatch);
      off += 2;
      if (lane < nb) out.put(off + lane, static_cast<uint32_t>(shr64(lmin, 8u * (nb - 1u - lane))));
      off += nb;
      put_packed(out.p + off, sh.red[warp], n, bits);
      put_packed(out.p + off + aligned_bytes(n, bits), sh.list[warp], npatch, w2);
      return;
    }
    // DELTA: base and first step as varints, then the further steps unless they are all the same
    const uint64_t zz = zigzag(second - first);
    const uint32_t l1 = varint_len(first), l2 = varint_len(zz);
    if (lane < l1) out.put(off + lane, varint_byte(first, lane, l1));
    else if (lane < l1 + l2) out.put(off + lane, varint_byte(zz, lane - l1, l2));
    if (kind == kDeltaFixed) return;
    uint64_t d[4], x[4], last = 0;
#pragma unroll
    for (uint32_t q = 0; q < 4; q++) {
      uint64_t prev = shfl_up64(v[q], 1);
      if (lane == 0) prev = last;
      last = shfl64(v[q], 31);
      d[q] = v[q] - prev;
    }
#pragma unroll
    for (uint32_t q = 0; q < 4; q++) {  // element i is the step to value i + 2
      const uint64_t here = shfl64(d[q], (lane + 2u) & 31u);
      const uint64_t next = q < 3 ? shfl64(d[q + 1], (lane + 2u) & 31u) : 0ull;
      x[q] = lane < 30u ? here : next;
    }
    put_aligned(out.p + off + l1 + l2, x[0], x[1], x[2], x[3], n - 2u, bits);
  }

  static __device__ __forceinline__ uint32_t measure(const T* val, uint32_t n, bool run, Shared& sh, uint32_t item,
                                                     uint32_t warp, uint32_t lane) {
    ItemV2 it;
    it.load(val, n, lane);
    it.choose(run, sh, warp, lane);
    if (lane == 0) sh.how[item] = it.pack();
    return it.size;
  }
  static __device__ __forceinline__ void write(const T* val, uint32_t n, bool, const Bytes& out, Shared& sh, uint32_t item,
                                               uint32_t warp, uint32_t lane) {
    ItemV2 it;
    it.load(val, n, lane);
    it.unpack(sh.how[item]);
    it.put_item(out, 0, sh, warp, lane);
  }
};

// Front warps: the tile whose first value is t0.
template <bool V1, typename T, class S, class Get>
__device__ __forceinline__ void prepare_tile(EncodeTile<T, S>& t, const Get& get, uint64_t t0, uint64_t n, uint32_t warp,
                                             uint32_t lane) {
  constexpr uint32_t kTile = S::kTile, kAhead = S::kAhead, kMaskWords = S::kMaskWords, FRONT = S::kFront;
  const uint32_t end = static_cast<uint32_t>(n - t0 < kTile + kAhead ? n - t0 : kTile + kAhead);
  constexpr uint32_t kStep = 32 * FRONT;
  for (uint32_t i = 32u * warp + lane; i < end; i += 8 * kStep) {
    T x[8];  // several loads in flight
#pragma unroll
    for (uint32_t k = 0; k < 8; k++)
      if (i + k * kStep < end) x[k] = static_cast<T>(get(t0 + i + k * kStep));
#pragma unroll
    for (uint32_t k = 0; k < 8; k++)
      if (i + k * kStep < end) t.val[i + k * kStep] = x[k];
  }
  group_barrier<1, FRONT>();
#pragma unroll 2
  for (uint32_t w = warp; w < kMaskWords; w += FRONT) {  // comparisons of values t0 + j
    const uint32_t j = 32u * w + lane;
    bool pa = false, pb = false;
    if constexpr (V1) {
      if (j + 2u < end) {
        const T x0 = t.val[j], x1 = t.val[j + 1], x2 = t.val[j + 2];
        const int64_t d = step_of<T>(x0, x1);
        pb = d == step_of<T>(x1, x2);
        pa = pb && d >= -128 && d <= 127;
      }
    } else {
      if (j >= 1u && j < end) {
        pb = t.val[j] == t.val[j - 1];
        pa = pb && j >= 2u && t.val[j - 1] == t.val[j - 2];
      }
    }
    const uint32_t ma = __ballot_sync(FULL, pa), mb = __ballot_sync(FULL, pb);
    if (lane == 0) {
      t.a[w] = ma;
      t.b[w] = mb;
    }
  }
  group_barrier<1, FRONT>();
  for (uint32_t w = warp; w < kTile / 32u; w += FRONT) {  // the item that would start at p
    const uint32_t p = 32u * w + lane, left = p < end ? end - p : 0u;
    uint32_t len, run;
    if constexpr (V1) {
      const uint32_t r = distance_to_set(t.a, 0u, w, 0, lane), z = distance_to_set(t.b, FULL, w, 0, lane) + 2u;
      run = r == 0u;
      len = run ? (z < 129u ? z : 129u) : (r < 127u ? r : 127u);
    } else {
      const uint32_t r = distance_to_set(t.a, 0u, w, 2, lane), z = distance_to_set(t.b, FULL, w, 1, lane) + 1u;
      run = r == 0u;
      len = run ? (z < 128u ? z : 128u) : (r < 126u ? r : 128u);
    }
    t.len[p] = static_cast<uint16_t>((len < left ? len : left) | (run << 8));
  }
  group_barrier<1, FRONT>();
  if (warp != 0 || lane != 0) return;
  uint32_t p = 0, items = 0;  // items that start in the tile
  while (p < kTile && p < end) {
    const uint32_t v = t.len[p];
    t.item[items++] = p | (v << 12);
    p += v & 0xffu;
  }
  t.items = items;
  t.next = t0 + p;
}

// One CTA per chunk.  Bound by the latency of the front's walk and of the back's longest items, with small chunks by
// how many fit the GPU at once.
template <class Item, typename T, bool V1>
__global__ void __launch_bounds__(Item::Shared::kThreads, Item::Shared::kCtas)
    k_encode(const uint8_t* __restrict__ in, uint64_t in_bytes, uint64_t chunk_bytes, uint8_t* __restrict__ scratch,
             uint64_t slot, uint64_t* __restrict__ lens) {
  constexpr bool kAlone = Item::Shared::kAlone;
  constexpr uint32_t kFront = kAlone ? 0 : Item::Shared::kFront, kBack = Item::Shared::kBack;
  extern __shared__ __align__(16) uint8_t smem[];
  auto& sh = *reinterpret_cast<typename Item::Shared*>(smem);
  const uint32_t lane = threadIdx.x & 31u;
  const bool front = threadIdx.x < 32u * kFront;  // none where one warp does all
  const uint32_t warp = (threadIdx.x >> 5) - (front ? 0u : kFront);
  const uint64_t chunk = blockIdx.x;
  const uint64_t n = chunk_bytes / sizeof(T);
  using W = typename Wide<T>::T;
  const PaddedChunk<W> get{in, in_bytes, chunk * chunk_bytes};
  uint8_t* out = scratch + chunk * slot;
  uint64_t base = 0, ready = 0;  // bytes written; first value of the tile to prepare
  bool have = false;             // the back has a tile
  if (threadIdx.x < 4) sh.taken[threadIdx.x >> 1][threadIdx.x & 1u] = 0;
  __syncthreads();
  for (uint32_t c = 0; ready < n || have; c ^= 1u) {
    if (front || kAlone) {
      if (ready < n) prepare_tile<V1, T>(sh.tile[kAlone ? 0 : c], get, ready, n, warp, lane);
      __syncwarp();
    }
    if (kAlone || (!front && have)) {
      const typename Item::Tile& t = sh.tile[kAlone ? 0 : c ^ 1u];
      const uint32_t items = t.items;
      // RLE v2 items take from 50 to some 600 instructions, so the warps take them as they come (1064 us with
      // every kBack-th for each warp, 1032 with the measuring as they come, 932 with the writing, too); RLE v1
      // items are too short for that (127 | 133)
      const auto next = [&](uint32_t i, uint32_t* taken) {
        if (V1) return i + kBack;
        uint32_t k = 0;
        if (lane == 0) k = atomicAdd(taken, 1u);
        return __shfl_sync(FULL, k, 0);
      };
      for (uint32_t i = V1 ? warp : next(0, &sh.taken[c][0]); i < items; i = next(i, &sh.taken[c][0])) {
        const uint32_t d = t.item[i];
        const uint32_t size = Item::measure(t.val + (d & 0xfffu), (d >> 12) & 0xffu, (d >> 20) != 0, sh, i, warp, lane);
        if (lane == 0) sh.off[i] = size;
      }
      group_barrier<2, kBack>();
      // every warp sums its share of the items, then starts from the sums of the warps below
      const uint32_t per = (items + kBack - 1u) / kBack, i0 = warp * per < items ? warp * per : items;
      const uint32_t i1 = i0 + per < items ? i0 + per : items;
      uint32_t sum = 0;
      for (uint32_t i = i0 + lane; i < i1; i += 32) sum += sh.off[i];
      sum = __reduce_add_sync(FULL, sum);
      if (lane == 0) sh.part[warp] = sum;
      group_barrier<2, kBack>();
      const uint32_t mine = lane < kBack ? sh.part[lane] : 0u;
      uint32_t at = __reduce_add_sync(FULL, lane < warp ? mine : 0u);
      const uint32_t total = __reduce_add_sync(FULL, mine);
      const auto write = [&](uint32_t i, uint32_t at, uint32_t size) {
        const uint32_t d = t.item[i];
        if (base + at + size <= slot)  // else the stream's length will say that it did not fit
          Item::write(t.val + (d & 0xfffu), (d >> 12) & 0xffu, (d >> 20) != 0, Bytes{out + base + at}, sh, i, warp, lane);
      };
      if (V1) {
        for (uint32_t i = i0; i < i1; i++) {
          const uint32_t size = sh.off[i];
          write(i, at, size);
          at += size;
        }
      } else {
        for (uint32_t i = i0; i < i1; i += 32) {
          const uint32_t size = i + lane < i1 ? sh.off[i + lane] : 0u, upto = scan_add(size, lane);
          if (i + lane < i1) sh.end[i + lane] = at + upto;
          at += __shfl_sync(FULL, upto, 31);
        }
        if (threadIdx.x == 32u * kFront) sh.taken[c ^ 1u][0] = sh.taken[c ^ 1u][1] = 0;
        group_barrier<2, kBack>();
        for (uint32_t i = next(0, &sh.taken[c][1]); i < items; i = next(i, &sh.taken[c][1]))
          write(i, sh.end[i] - sh.off[i], sh.off[i]);
      }
      base += total;
    }
    __syncthreads();
    have = ready < n && !kAlone;
    if (ready < n) ready = sh.tile[kAlone ? 0 : c].next;
    if (kAlone) __syncwarp();
  }
  if (threadIdx.x == 32u * kFront) lens[chunk] = base > slot ? kOverflow : base;
}

template <uint64_t ALIGN>
__device__ __forceinline__ uint64_t round_up(uint64_t len) {
  return (len + ALIGN - 1) / ALIGN * ALIGN;
}

// blk_off[i] = sum of round_up(lens[k], ALIGN) for k < i, and blk_off[n] = the total or, for RLE v2,
// the original size (encoder_trans.h:545); one CTA of 1024 threads, each summing a contiguous range.
template <uint64_t ALIGN, bool LAST_IS_SIZE>
__global__ void __launch_bounds__(1024) k_scan_offsets(const uint64_t* __restrict__ lens, uint64_t n, uint64_t in_bytes,
                                                       uint64_t* __restrict__ blk_off, int32_t* __restrict__ status) {
  __shared__ uint64_t part[32];
  const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
  const uint64_t per = (n + 1023) / 1024, a = t * per < n ? t * per : n, b = a + per < n ? a + per : n;
  uint64_t s = 0;
  bool over = false;
  for (uint64_t i = a; i < b; i++) {
    over |= lens[i] == kOverflow;
    s += round_up<ALIGN>(lens[i]);
  }
  const uint64_t upto = warp_scan_add64(s, lane);
  if (lane == 31) part[warp] = upto;
  const int bad = __syncthreads_or(over);
  const uint64_t below = warp_scan_add64(part[lane], lane);  // of the warps up to `lane`
  uint64_t run = upto - s + (warp ? shfl64(below, static_cast<int>(warp) - 1) : 0);
  for (uint64_t i = a; i < b; i++) {
    blk_off[i] = run;
    run += round_up<ALIGN>(lens[i]);
  }
  const uint64_t total = shfl64(below, 31);
  if (t == 0) {
    blk_off[n] = LAST_IS_SIZE ? in_bytes : total;
    if (status) *status = bad ? CODAG_ECORRUPT : CODAG_OK;
  }
}

// Stream i = blockIdx.x, or one of gridDim.y shares of it, goes to out + head + blk_off[i] and is zero
// padded to ALIGN bytes.  RLE v1 (head 8): the blob starts with the original size.
template <uint64_t ALIGN, uint32_t HEAD>
__global__ void __launch_bounds__(256) k_gather(const uint8_t* __restrict__ scratch, uint64_t slot,
                                                const uint64_t* __restrict__ lens, uint64_t n, uint8_t* __restrict__ out,
                                                uint64_t capacity, const uint64_t* __restrict__ blk_off,
                                                uint64_t* __restrict__ col_len, uint64_t in_bytes,
                                                uint64_t* __restrict__ out_bytes, int32_t* __restrict__ status) {
  const uint64_t total = HEAD + blk_off[n - 1] + round_up<ALIGN>(lens[n - 1]);
  const uint64_t i = blockIdx.x;
  const bool first = threadIdx.x == 0 && blockIdx.y == 0;
  if (first && i == 0) {
    if (out_bytes) *out_bytes = total;
    if (total > capacity && status) *status = CODAG_ELIMIT;
    if (HEAD == 8 && capacity >= 8) *reinterpret_cast<uint64_t*>(out) = in_bytes;
  }
  if (total > capacity) return;
  const uint64_t len = lens[i], off = HEAD + blk_off[i];
  if (first) col_len[i] = len;
  if (len == kOverflow) return;
  const uint64_t words = round_up<ALIGN>(len) / 4, full = len / 4;
  const uint32_t* src = reinterpret_cast<const uint32_t*>(scratch + i * slot);
  uint32_t* dst = reinterpret_cast<uint32_t*>(out + off);  // 4-byte aligned: HEAD, ALIGN multiples of 4
  const uint64_t share = (words + gridDim.y - 1) / gridDim.y, w0 = blockIdx.y * share;
  const uint64_t w1 = w0 + share < words ? w0 + share : words, wf = w1 < full ? w1 : full;
#pragma unroll 4
  for (uint64_t w = w0 + threadIdx.x; w < wf; w += 256) dst[w] = src[w];
  for (uint64_t w = (w0 > full ? w0 : full) + threadIdx.x; w < w1; w += 256) {
    const uint64_t b0 = 4 * w;  // keep the stream's bytes, zero the padding
    dst[w] = b0 < len ? src[w] & ((1u << (8 * (len - b0))) - 1u) : 0u;
  }
}

bool valid_elem(int e) { return e == 1 || e == 2 || e == 4 || e == 8; }

uint64_t chunks_of(uint64_t in_bytes, uint64_t chunk_bytes) {
  return (in_bytes + chunk_bytes * 32 - 1) / (chunk_bytes * 32) * 32;  // rlev1.h:111-112, encoder_trans.h:490
}

// Workspace slot per chunk: the longest stream a chunk can give, 16-byte aligned.  RLE v1: every
// value a varint of ceil(8E/7) bytes plus a header per 127 literals; RLE v2: at most 1.25x the
// input for 64-bit values, taken as 2x plus a margin for every width.
uint64_t slot_of(int codec, uint64_t chunk_bytes, int e) {
  const uint64_t cnt = chunk_bytes / static_cast<uint64_t>(e);
  const uint64_t b = codec == CODAG_CODEC_RLEV1 ? cnt * ((8u * e + 6u) / 7u) + cnt / 127u + 64u : 2u * chunk_bytes + 4096u;
  return (b + 15u) / 16u * 16u;
}

template <class Item, typename T, bool V1>
bool launch_shape(const uint8_t* in, uint64_t in_bytes, uint64_t chunk, uint64_t n, uint8_t* scratch, uint64_t slot,
                  uint64_t* lens, cudaStream_t s) {
  auto kern = k_encode<Item, T, V1>;
  constexpr uint32_t bytes = sizeof(typename Item::Shared);
  if (codag_capi::allow_smem(kern, bytes) != cudaSuccess) return false;
  kern<<<static_cast<unsigned>(n), Item::Shared::kThreads, bytes, s>>>(in, in_bytes, chunk, scratch, slot, lens);
  return true;
}

template <int CODEC, typename T>
bool launch_encode(const uint8_t* in, uint64_t in_bytes, uint64_t chunk, uint64_t n, uint8_t* scratch, uint64_t slot,
                   uint64_t* lens, cudaStream_t s) {
  constexpr bool V1 = CODEC == CODAG_CODEC_RLEV1;
  using Big = std::conditional_t<V1, ItemV1<T, BigV1>, ItemV2<T, BigV2>>;
  using One = std::conditional_t<V1, ItemV1<T, Small>, ItemV2<T, Small>>;
  const auto launch = small_pays<V1>(n, chunk / sizeof(T)) ? launch_shape<One, T, V1> : launch_shape<Big, T, V1>;
  return launch(in, in_bytes, chunk, n, scratch, slot, lens, s);
}

template <int CODEC>
codag_status compress(const uint8_t* d_in, uint64_t in_bytes, uint64_t chunk, int e, uint8_t* d_out, uint64_t capacity,
                      uint64_t* d_blk_off, uint64_t* d_col_len, uint64_t* d_out_bytes, int32_t* d_status, void* ws,
                      uint64_t ws_bytes, cudaStream_t s) {
  if (!d_in || !d_out || !d_blk_off || !d_col_len || !valid_elem(e) || chunk == 0 || chunk % e || in_bytes == 0 ||
      chunk >= (1ull << 31) || (reinterpret_cast<uintptr_t>(d_in) % e) || (reinterpret_cast<uintptr_t>(d_out) & 15u))
    return CODAG_EINVAL;
  if (CODEC == CODAG_CODEC_RLEV1 && chunk / e < 2) return CODAG_EINVAL;
  const uint64_t n = chunks_of(in_bytes, chunk), slot = slot_of(CODEC, chunk, e);
  if (!ws || ws_bytes < codag_compress_workspace_bytes(CODEC, in_bytes, chunk, e) ||
      (reinterpret_cast<uintptr_t>(ws) & 255u))
    return CODAG_EINVAL;
  (void)cudaGetLastError();  // an error earlier work left pending is not this call's
  uint8_t* scratch = static_cast<uint8_t*>(ws);
  uint64_t* lens = reinterpret_cast<uint64_t*>(scratch + n * slot);
  bool ok;
  switch (e) {
    case 8: ok = launch_encode<CODEC, uint64_t>(d_in, in_bytes, chunk, n, scratch, slot, lens, s); break;
    case 4: ok = launch_encode<CODEC, uint32_t>(d_in, in_bytes, chunk, n, scratch, slot, lens, s); break;
    case 2: ok = launch_encode<CODEC, uint16_t>(d_in, in_bytes, chunk, n, scratch, slot, lens, s); break;
    default: ok = launch_encode<CODEC, uint8_t>(d_in, in_bytes, chunk, n, scratch, slot, lens, s); break;
  }
  if (!ok) return CODAG_ECUDA;
  constexpr uint64_t A = CODEC == CODAG_CODEC_RLEV1 ? 4 : 128;  // encoder.h:780-783 / encoder_trans.h:352
  constexpr uint32_t H = CODEC == CODAG_CODEC_RLEV1 ? 8 : 0;    // rlev1.h:103-192: [u64 size][streams]
  constexpr bool V2 = CODEC == CODAG_CODEC_RLEV2;
  k_scan_offsets<A, V2><<<1, 1024, 0, s>>>(lens, n, in_bytes, d_blk_off, d_status);
  // eight CTAs a chunk where one each would leave SMs idle
  k_gather<A, H><<<dim3(static_cast<unsigned>(n), n < 1024 ? 8 : 1), 256, 0, s>>>(
      scratch, slot, lens, n, d_out, capacity, d_blk_off, d_col_len, in_bytes, d_out_bytes, d_status);
  return cudaGetLastError() == cudaSuccess ? CODAG_OK : CODAG_ECUDA;
}

}  // namespace

extern "C" uint64_t codag_compress_chunks(uint64_t in_bytes, uint64_t chunk_bytes) {
  return chunk_bytes ? chunks_of(in_bytes, chunk_bytes) : 0;
}

extern "C" uint64_t codag_compress_workspace_bytes(int codec, uint64_t in_bytes, uint64_t chunk_bytes, int elem_bytes) {
  if ((codec != CODAG_CODEC_RLEV1 && codec != CODAG_CODEC_RLEV2) || !valid_elem(elem_bytes) || !chunk_bytes) return 0;
  const uint64_t n = chunks_of(in_bytes, chunk_bytes);
  return n * slot_of(codec, chunk_bytes, elem_bytes) + n * 8;
}

extern "C" uint64_t codag_compress_bound(int codec, uint64_t in_bytes, uint64_t chunk_bytes, int elem_bytes) {
  if ((codec != CODAG_CODEC_RLEV1 && codec != CODAG_CODEC_RLEV2) || !valid_elem(elem_bytes) || !chunk_bytes) return 0;
  const uint64_t n = chunks_of(in_bytes, chunk_bytes), slot = slot_of(codec, chunk_bytes, elem_bytes);
  return codec == CODAG_CODEC_RLEV1 ? 8 + n * ((slot + 3) / 4 * 4) : n * ((slot + 127) / 128 * 128);
}

extern "C" codag_status codag_compress_rlev1(const uint8_t* d_in, uint64_t in_bytes, uint64_t chunk_bytes,
                                             int elem_bytes, uint8_t* d_blob, uint64_t blob_capacity,
                                             uint64_t* d_blk_off, uint64_t* d_col_len, uint64_t* d_blob_bytes,
                                             int32_t* d_status, void* d_workspace, uint64_t workspace_bytes,
                                             codag_stream_t stream) {
  return compress<CODAG_CODEC_RLEV1>(d_in, in_bytes, chunk_bytes, elem_bytes, d_blob, blob_capacity, d_blk_off,
                                     d_col_len, d_blob_bytes, d_status, d_workspace, workspace_bytes,
                                     reinterpret_cast<cudaStream_t>(stream));
}

extern "C" codag_status codag_compress_rlev2(const uint8_t* d_in, uint64_t in_bytes, uint64_t chunk_bytes,
                                             int elem_bytes, uint8_t* d_comp, uint64_t comp_capacity,
                                             uint64_t* d_blk_off, uint64_t* d_col_len, uint64_t* d_comp_bytes,
                                             int32_t* d_status, void* d_workspace, uint64_t workspace_bytes,
                                             codag_stream_t stream) {
  return compress<CODAG_CODEC_RLEV2>(d_in, in_bytes, chunk_bytes, elem_bytes, d_comp, comp_capacity, d_blk_off,
                                     d_col_len, d_comp_bytes, d_status, d_workspace, workspace_bytes,
                                     reinterpret_cast<cudaStream_t>(stream));
}
