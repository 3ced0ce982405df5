// Decoder of CODAG's transposed RLE v2 layout (include/codag.h, codag_decompress_rlev2_transposed).
//
// In that layout (include/rlev2/encoder_trans.h:8-182 and 359-391) a chunk is 32 substreams,
// substream t holding the values t*ru + k*32*ru + j (j < ru), and the chunk's bytes interleave
// the substreams in 4-byte words: word w of every substream longer than 4w, in substream
// order, then word w+1.  CODAG decodes it with one lane per substream fed by a reader warp
// through spin queues (include/rlev2/decoder_new.h:375-632, 1193-1230).  Here one warp
// decodes a chunk with no queue.  The set of substreams that still have a word w only shrinks
// as w grows, so it changes at most 32 times: the warp tabulates those segments of rows (first
// and last row, the mask of substreams present, the words before the segment; at most 32
// entries, 512 bytes of shared memory per warp), and lane t finds its word w at
// start + (w - first row) * popc(mask) + popc(mask & lanes below t) by itself.  Then every
// lane decodes its own substream and writes its values straight to their interleaved places
// in global memory.  The small table leaves occupancy to the registers, so many chunks' lanes
// wait on their word loads at once.  Where there are few chunks, four warps share one's substreams.
// 256 MiB of 64-bit values: 650 us with byte-wise headers and fields, 433 with a word at a time loaded when it
// was needed (a step from one value to the next took 600 cycles, most of it that load, which some lane or
// other does every time), 371 with the words copied to shared memory ahead of their use.  Header semantics are CODAG's (the oracle's restatement of
// decoder_new.h:1000-1184, quirks included: the uint8_t run length, the 32-bit patch mask, the
// arithmetic-shift zigzag and the DELTA direction taken from the base delta).
#include <cuda_runtime.h>

#include <cstdint>

#include "../../../include/codag.h"
#include "decode_rle.cuh"

using namespace codag_dev;

namespace {

// bytes of one lane's substream, read word by word from the interleaved region
// row segments of one chunk (shared memory): rows lo[s] <= w < hi[s] hold a word of exactly the
// substreams in mask[s], and words[s] words of the region come before row lo[s]
struct Segments {
  uint32_t hi[32], lo[32], mask[32], words[32];
};

constexpr uint32_t kWarps = 4;  // warps per block

constexpr uint32_t kFifo = 16;
struct LaneReader {
  const uint32_t* region;  // the chunk's region (128-byte aligned)
  const Segments* seg;
  uint32_t total;          // words in the region
  uint32_t lt;             // lanes below this one
  uint32_t len, words;     // substream bytes, and words
  uint32_t p;              // next byte
  uint32_t cw, cv;         // cached word index and value
  uint32_t s;              // segment of the last word loaded by start() (rows only grow, so it only moves forward)
  // The words to come, kFifo at most, are copied to the lane's column of shared memory ahead of their use.
  uint32_t fifo;           // word w at fifo + 128 * (w % kFifo)
  uint32_t issued = 0, avail = 0;  // words asked for, and known to be there
  uint32_t next_at = 0, next_step = 0, next_hi = 0, next_s = 0;  // place of word `issued`, as start() finds it
  bool bad = false;

  // Called by all lanes every few values: what was asked for last time is there by now, and the
  // next N words, kFifo at most behind `low`, the first one still needed, are asked for.
  template <uint32_t N>
  __device__ __forceinline__ void top_up(uint32_t low) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    avail = issued;
    if (issued < low) {
      issued = low;
      next_hi = 0;
    }
    const uint32_t lim = low + kFifo < words ? low + kFifo : words;
#pragma unroll 2
    for (uint32_t i = 0; i < N; i++) {
      if (issued < lim) {
        if (issued >= next_hi) {
          while (issued >= seg->hi[next_s]) next_s++;
          const uint32_t m = seg->mask[next_s];
          next_hi = seg->hi[next_s];
          next_step = __popc(m);
          next_at = seg->words[next_s] + (issued - seg->lo[next_s]) * next_step + __popc(m & lt);
        }
        if (next_at < total) {
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(fifo + 128u * (issued % kFifo)), "l"(region + next_at)
                       : "memory");
          issued++;
          next_at += next_step;
        }
      }
    }
  }
  __device__ __forceinline__ uint32_t ahead(uint32_t w) const { return ld_s32(fifo + 128u * (w % kFifo)); }
  __device__ __forceinline__ uint32_t word(uint32_t w) { return w < avail ? ahead(w) : __ldg(region + start(w)); }

  // where word w of this substream sits in the region; w < its word count <= the last
  // segment's hi keeps the walk inside the table, and the region has `total` words
  __device__ __forceinline__ uint32_t start(uint32_t w) {
    while (w >= seg->hi[s]) s++;
    const uint32_t m = seg->mask[s];
    const uint32_t at = seg->words[s] + (w - seg->lo[s]) * __popc(m) + __popc(m & lt);
    if (at >= total) {
      bad = true;
      return 0;
    }
    return at;
  }

  __device__ __forceinline__ uint32_t byte() {
    if (p >= len) {
      bad = true;
      return 0;
    }
    const uint32_t w = p >> 2;
    if (w != cw) {
      cw = w;
      cv = word(w);
    }
    return (cv >> (8u * (p++ & 3u))) & 0xffu;
  }

  // the 16 bytes from p on, least significant first; bytes past the substream's last word are 0
  __device__ __forceinline__ void window(uint32_t* l) {
    const uint32_t w = p >> 2, n = words - w;
    uint32_t x[5];
#pragma unroll
    for (uint32_t i = 0; i < 5; i++) x[i] = i < n ? ahead(w + i) : 0u;
    if (avail < (n < 5u ? words : w + 5u)) {  // not all there yet
      const uint32_t at = start(w), same = seg->hi[s] - w, step = __popc(seg->mask[s]);  // words of this row segment
      x[0] = __ldg(region + at);
#pragma unroll
      for (uint32_t i = 1; i < 5; i++) x[i] = i < n && i < same ? __ldg(region + at + i * step) : 0u;
      if (same < 5u && same < n) {  // the others lie in later segments
        const uint32_t s0 = s;
        for (uint32_t i = same; i < 5u && i < n; i++) {
          const uint32_t v = __ldg(region + start(w + i));
          if (i == 1) x[1] = v;
          else if (i == 2) x[2] = v;
          else if (i == 3) x[3] = v;
          else x[4] = v;
        }
        s = s0;
      }
    }
#pragma unroll
    for (uint32_t i = 0; i < 4; i++) l[i] = __funnelshift_r(x[i], x[i + 1], 8u * (p & 3u));
  }

  // MSB-first bit fields of the `total` bytes from p on (decoder_new.h:1024-1040), read through a 64-bit
  // buffer a word at a time; p moves past them at once
  uint64_t bb;   // bits not yet read, the next on top
  uint32_t bc;   // how many
  uint32_t bw;   // next word
  __device__ __forceinline__ void fields(uint32_t total) {
    if (total > len - p) {
      bad = true;
      return;
    }
    bb = 0;
    bc = 0;
    bw = p >> 2;
    if (total) {
      refill();
      bb <<= 8u * (p & 3u);
      bc -= 8u * (p & 3u);
    }
    p += total;
  }
  __device__ __forceinline__ void refill() {
    if (bw != cw) {
      cw = bw;
      cv = word(bw);
    }
    bb |= static_cast<uint64_t>(__byte_perm(cv, 0u, 0x0123u)) << (32u - bc);
    bc += 32;
    bw++;
  }
  __device__ __forceinline__ uint32_t field32(uint32_t n) {  // 1..32 bits
    if (bc < n) refill();
    const uint32_t v = static_cast<uint32_t>(bb >> (64u - n));
    bb <<= n;
    bc -= n;
    return v;
  }
  __device__ __forceinline__ uint64_t field(uint32_t n) {  // 1..64 bits
    if (n <= 32u) return field32(n);
    const uint64_t hi = field32(n - 32u);
    return (hi << 32) | field32(32);
  }
};

// value k of substream t lands on element t*ru + (k/ru)*32*ru + k%ru of the chunk
template <typename T>
struct LaneOut {
  T* chunk;
  uint32_t t, ru, cap, store;  // cap: values per substream; store: elements of the chunk to store
  uint32_t n;
  uint32_t e, j;  // element of value n, and n % ru (stepped without a division)
  bool over;
  __device__ __forceinline__ uint32_t elem(uint32_t k) const { return t * ru + (k / ru) * 32u * ru + k % ru; }
  __device__ __forceinline__ void put(uint64_t v) {
    if (n >= cap) {
      over = true;
      return;
    }
    if (e < store) chunk[e] = static_cast<T>(v);
    n++;
    if (++j == ru) {  // next group of ru values, 32 * ru elements on
      j = 0;
      e += 31u * ru + 1u;
    } else {
      e++;
    }
  }
  __device__ __forceinline__ uint64_t get(uint32_t k) const {
    const uint32_t e = elem(k);
    return e < store ? static_cast<uint64_t>(chunk[e]) : 0ull;
  }
  __device__ __forceinline__ void set(uint32_t k, uint64_t v) {
    const uint32_t e = elem(k);
    if (e < store) chunk[e] = static_cast<T>(v);
  }
};

__device__ __noinline__ uint64_t uvarint(LaneReader& r) {
  uint64_t v = 0;
  uint32_t off = 0, b;
  do {
    b = r.byte();
    if (r.bad) return 0;
    v |= shl64(b & 0x7fu, off);
    off += 7;
  } while (b >= 0x80u);
  return v;
}

// One lane's substream as a state machine that yields one value per pass (four where values are narrow): a lane
// whose run has ended reads its next header first, so the warp's lanes meet again after a value or four
// instead of waiting for the longest run among them.  2048 chunks, one | two | four values a pass: 64 bits
// 452 us | 468 | 479, 32 bits 864 | 864 | 880, 16 bits 1615 | 1603 | 1521, 8 bits 2997 | 3097 | 2826 (before the words
// came ahead of their use; 371, 723, 1202 and 2379 now).
// Every run kind yields its next value by one step, x = v + d or v - d (v kept as x for the kinds that
// accumulate), d being the run's next bit field or a constant, so the only fork inside the
// step is whether the lane reads bits.
constexpr int kEnd = -1;

template <typename T>
__device__ int decode_substream(LaneReader& r, LaneOut<T>& o, bool go) {
  constexpr uint64_t M = sizeof(T) == 8 ? ~0ull : ((1ull << (8 * sizeof(T))) - 1ull);
  constexpr int kValues = sizeof(T) <= 2 ? 4 : 1;
  uint32_t rem = 0, fbw = 0;
  uint64_t v = 0, bd = 0;  // repeat: the value; delta: running value and base delta; patched: base
  bool bits = false, acc = false, sub = false, patched = false;
  uint32_t pw = 0, pgw = 0, pll = 0, base_out = 0;  // patched: patch width, gap width, list length
  int st = CODAG_OK;
  // 64-bit values take at most two words each, so a top-up every kPasses passes keeps ahead of them.
  constexpr uint32_t kPasses = kValues == 1 ? 4 : 1, kTopUp = kValues == 1 ? 8 : 4;
  uint32_t pass = 0;
  r.template top_up<kFifo>(0);
  const auto header = [&]() -> int {  // the next header with values; kEnd at the end of the substream
    for (;;) {
      if (patched) {  // the run's values are out: patch them (decoder_new.h:1166-1183)
        if (pw + pgw > 64) return CODAG_ECORRUPT;
        const uint64_t pmask = pw >= 32 ? 0xFFFFFFFFull : ((1ull << pw) - 1ull);  // 32-bit mask (:1103)
        const uint32_t cfb = v2_closest(pw + pgw);
        r.fields((pll * cfb + 7u) / 8u);
        if (r.bad) return CODAG_ECORRUPT;
        uint64_t gap = 0;
        while (pll-- > 0) {
          const uint64_t ent = r.field(cfb);
          gap += shr64(ent, pw);
          const uint64_t idx = base_out + gap;
          if (idx >= o.n) return CODAG_ECORRUPT;
          const uint64_t patch = shl64((ent & pmask) & M, fbw) & M;
          const uint64_t x = o.get(static_cast<uint32_t>(idx));
          o.set(static_cast<uint32_t>(idx), ((((x - v) & M) | patch) + v) & M);
        }
      }
      patched = false;
      if (r.p >= r.len) return kEnd;
      // every kind from the same 16 bytes, so that lanes at different kinds go together
      uint32_t l[4];
      r.window(l);
      const uint64_t x0 = (static_cast<uint64_t>(l[1]) << 32) | l[0], x8 = (static_cast<uint64_t>(l[3]) << 32) | l[2];
      const uint32_t first = l[0] & 0xffu, kind = first >> 6, enc = (first >> 1) & 0x1fu;
      const uint32_t third = (l[0] >> 16) & 0xffu, fourth = l[0] >> 24;
      const uint32_t len8 = ((((first & 1u) << 8) | ((l[0] >> 8) & 0xffu)) + 1u) & 0xffu;  // a uint8_t length (:1018)
      // SHORT_REPEAT's value (decoder_new.h:1004-1014) after 1 byte, PATCHED_BASE's base (:1092-1165) after 4: 1 to 8
      // bytes, big-endian
      const uint32_t lead = kind == 0 ? 1u : 4u, nb = (kind == 0 ? (first >> 3) & 7u : (third >> 5) & 7u) + 1u;
      const uint64_t big = bswap64((x0 >> (8u * lead)) | (x8 << (64u - 8u * lead))) >> (64u - 8u * nb);
      uint32_t bytes = kind & 1u ? 2u : lead + nb;
      fbw = v2_width(enc);
      rem = len8;
      v = kind & 1u ? 0 : big;
      bd = 0;
      bits = kind != 0;
      acc = kind == 0 || kind == 3;
      sub = false;
      if (kind == 0) {
        rem = (first & 7u) + 3u;
        v &= M;
      }
      patched = kind == 2;
      if (patched) {
        pw = v2_width(third & 0x1fu);
        pgw = ((fourth >> 5) & 7u) + 1u;
        pll = fourth & 0x1fu;
        base_out = o.n;
      }
      if (kind == 3) {  // DELTA (decoder_new.h:1044-1091): base and base delta as varints
        const uint64_t lo = (x0 >> 16) | (x8 << 48), ends = ~lo & 0x8080808080808080ull, second = ends & (ends - 1ull);
        uint64_t u;
        if (second) {  // both within 8 bytes
          const uint32_t l1 = (ctz64(ends) >> 3) + 1u, l12 = (ctz64(second) >> 3) + 1u;
          v = leb_compact(lo, l1);
          u = leb_compact(lo >> (8u * l1), l12 - l1);
          bytes += l12;
        } else {
          LaneReader t = r;  // a copy, so that the reader itself stays in registers
          t.p += 2;
          v = uvarint(t);
          u = uvarint(t);
          if (t.bad) return CODAG_ECORRUPT;
          bytes = t.p - r.p;
        }
        v &= M;
        const int64_t t = static_cast<int64_t>(u);
        bd = static_cast<uint64_t>((t >> 1) ^ -(t & 1)) & M;  // arithmetic shift (:990)
        rem = (len8 - 2u) & 0xffu;
        bits = enc != 0;        // else every step adds the base delta
        sub = bits && bd == 0;  // multiplier = base_delta > 0 ? 1 : -1 on the unsigned type (:1057)
      }
      if (bytes > r.len - r.p) return CODAG_ECORRUPT;
      r.p += bytes;
      if (kind == 3) {
        o.put(v);
        v = (v + bd) & M;
        o.put(v);
      }
      if (bits && !r.bad) r.fields((rem * fbw + 7u) / 8u);
      if (r.bad || o.over) return CODAG_ECORRUPT;
      if (rem) return CODAG_OK;
    }
  };
  while (__any_sync(FULL, go)) {
    if (pass++ % kPasses == 0) {
      // a run's last word can be the next header's first
      r.template top_up<kTopUp>(!go ? r.words : bits && rem ? r.bw - 1u : r.p >> 2);
    }
    if (go && rem == 0) {
      st = header();
      go = st == CODAG_OK;
    }
    __syncwarp();
#pragma unroll 1
    for (int b = 0; b < kValues; b++) {
      if (go && rem) {
        const uint64_t d = bits ? r.field(fbw) & M : bd;
        const uint64_t x = (sub ? v - d : v + d) & M;
        if (acc) v = x;
        o.put(x);
        rem--;
        if (o.over) {
          st = CODAG_ECORRUPT;
          go = false;
        }
      }
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  return st == kEnd ? CODAG_OK : st;
}

// values of substream t whose elements fall below `store`
__device__ __forceinline__ uint32_t needed(uint32_t t, uint32_t ru, uint32_t store) {
  const uint32_t grp = 32u * ru, g = store / grp, rem = store % grp;
  const uint32_t lo = t * ru;
  return g * ru + (rem > lo ? (rem - lo < ru ? rem - lo : ru) : 0u);
}

// SPLIT warps share a chunk
template <typename T, uint32_t SPLIT>
__global__ void __launch_bounds__(32 * kWarps)
    k_rlev2_transposed(const uint8_t* __restrict__ comp, uint64_t comp_bytes, const uint64_t* __restrict__ blk_off,
                       const uint64_t* __restrict__ col_len, uint64_t n_chunks, uint64_t chunk_bytes, uint32_t ru,
                       uint8_t* __restrict__ out, uint64_t out_bytes, int32_t* __restrict__ status,
                       uint32_t max_words) {
  __shared__ Segments segs[kWarps];
  __shared__ uint32_t fifos[kWarps][kFifo][32];
  __shared__ uint32_t part[kWarps];  // the warps' statuses
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint64_t c = (static_cast<uint64_t>(blockIdx.x) * kWarps + warp) / SPLIT;
  const bool real = c < n_chunks;
  Segments* seg = segs + warp;
  const uint64_t len64 = real ? col_len[32 * c + lane] : 0;
  const uint32_t words = static_cast<uint32_t>(len64 < (1ull << 34) ? (len64 + 3) / 4 : 0xffffffffu);
  const uint32_t maxw = __reduce_max_sync(FULL, words);
  const uint64_t total = 4ull * __reduce_add_sync(FULL, words);
  const uint64_t off = real ? blk_off[c] : 0;
  int st = CODAG_OK;
  if (maxw > max_words || (off & 3u) || off > comp_bytes || total > comp_bytes - off) st = CODAG_ECORRUPT;
  const uint64_t base_e = c * (chunk_bytes / sizeof(T));
  const uint64_t store_b = c * chunk_bytes < out_bytes ? (out_bytes - c * chunk_bytes < chunk_bytes
                                                             ? out_bytes - c * chunk_bytes : chunk_bytes) : 0;
  const uint32_t store = static_cast<uint32_t>(store_b / sizeof(T));
  if (st == CODAG_OK && real) {
    // one segment per distinct word count: each pass drops at least one substream, so at most 32
    uint32_t run = 0, row = 0, ns = 0;
    for (uint32_t m = __ballot_sync(FULL, words > 0); m; m = __ballot_sync(FULL, words > row)) {
      const uint32_t nxt = __reduce_min_sync(FULL, words > row ? words : 0xffffffffu);
      if (lane == 0) {
        seg->hi[ns] = nxt;
        seg->lo[ns] = row;
        seg->mask[ns] = m;
        seg->words[ns] = run;
      }
      run += (nxt - row) * __popc(m);
      row = nxt;
      ns++;
    }
    __syncwarp();
    // this warp's substreams, one for each of the first lanes
    constexpr uint32_t kLanes = 32u / SPLIT;
    const bool mine = lane < kLanes;
    const uint32_t t = SPLIT == 1 ? lane : (warp % SPLIT) * kLanes + lane % kLanes;
    LaneReader r{reinterpret_cast<const uint32_t*>(comp + off), seg, run, (1u << t) - 1u,
                 __shfl_sync(FULL, static_cast<uint32_t>(len64), t), __shfl_sync(FULL, words, t), 0, 0xffffffffu, 0, 0,
                 smem_u32(&fifos[warp][0][lane])};
    LaneOut<T> o{reinterpret_cast<T*>(out) + base_e, t, ru,
                 static_cast<uint32_t>(chunk_bytes / sizeof(T) / 32), store, 0, t * ru, 0, false};
    int s = decode_substream<T>(r, o, mine);
    if (s == CODAG_OK && mine && o.n < needed(t, ru, store)) s = CODAG_ECORRUPT;
    st = __reduce_max_sync(FULL, static_cast<uint32_t>(s));
  }
  if (SPLIT > 1) {
    if (lane == 0) part[warp] = static_cast<uint32_t>(st);
    __syncthreads();
    if (lane < SPLIT) st = max(st, static_cast<int>(part[warp / SPLIT * SPLIT + lane]));
    st = __reduce_max_sync(FULL, static_cast<uint32_t>(st));
  }
  if (status && real && lane == 0 && warp % SPLIT == 0) status[c] = st;
}

// Up to how many chunks four warps with eight substreams each are faster than one with all 32: with fewer
// lanes a pass meets fewer headers, at the price of issue slots.  Measured, us, one | four warps, 64-bit
// values: 300 chunks 300 | 249, 592 306 | 298, 900 317 | 387; 32 bits 604 | 502, 609 | 572, 635 | 741.  Narrow values
// gain nothing (16 bits, 300 chunks: 957 | 951), nor do two warps of sixteen over the better of the others.
constexpr uint64_t kFewChunks = 4 * 148;

bool valid_elem(int e) { return e == 1 || e == 2 || e == 4 || e == 8; }

template <typename T>
codag_status launch(const uint8_t* comp, uint64_t comp_bytes, const uint64_t* blk_off, const uint64_t* col_len,
                    uint64_t n, uint64_t chunk, uint32_t ru, uint8_t* out, uint64_t out_bytes, int32_t* status,
                    cudaStream_t s) {
  // a substream is at most about twice its share of the chunk (the encoders' bound), in words
  const uint32_t max_words = static_cast<uint32_t>((chunk / 32 * 2 + 1024) / 4);
  constexpr uint32_t kSplit = sizeof(T) >= 4 ? 4 : 1;
  const bool few = n <= kFewChunks;
  const uint64_t grid = (n * (few ? kSplit : 1u) + kWarps - 1) / kWarps;
  if (grid > 0x7fffffffull) return CODAG_EINVAL;
  auto kern = few ? k_rlev2_transposed<T, kSplit> : k_rlev2_transposed<T, 1>;
  kern<<<static_cast<unsigned>(grid), 32 * kWarps, 0, s>>>(comp, comp_bytes, blk_off, col_len, n, chunk, ru, out, out_bytes,
                                                           status, max_words);
  return cudaGetLastError() == cudaSuccess ? CODAG_OK : CODAG_ECUDA;
}

}  // namespace

extern "C" codag_status codag_decompress_rlev2_transposed(const uint8_t* d_comp, uint64_t comp_bytes,
                                                          const uint64_t* d_blk_off, const uint64_t* d_col_len,
                                                          uint64_t n_chunks, uint64_t chunk_bytes, int elem_bytes,
                                                          int read_unit, uint8_t* d_out, uint64_t out_bytes,
                                                          int32_t* d_chunk_status, codag_stream_t stream) {
  if (!d_comp || !d_blk_off || !d_col_len || (!d_out && out_bytes) || !valid_elem(elem_bytes) || read_unit <= 0 ||
      chunk_bytes == 0 || chunk_bytes >= (1ull << 31) ||
      chunk_bytes % (32ull * static_cast<uint64_t>(read_unit) * static_cast<uint64_t>(elem_bytes)) ||
      (reinterpret_cast<uintptr_t>(d_out) % elem_bytes) || (reinterpret_cast<uintptr_t>(d_comp) & 3u))
    return CODAG_EINVAL;
  if (n_chunks == 0) return CODAG_OK;
  (void)cudaGetLastError();  // an error earlier work left pending is not this call's
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const uint32_t ru = static_cast<uint32_t>(read_unit);
  switch (elem_bytes) {
    case 8: return launch<uint64_t>(d_comp, comp_bytes, d_blk_off, d_col_len, n_chunks, chunk_bytes, ru, d_out, out_bytes, d_chunk_status, s);
    case 4: return launch<uint32_t>(d_comp, comp_bytes, d_blk_off, d_col_len, n_chunks, chunk_bytes, ru, d_out, out_bytes, d_chunk_status, s);
    case 2: return launch<uint16_t>(d_comp, comp_bytes, d_blk_off, d_col_len, n_chunks, chunk_bytes, ru, d_out, out_bytes, d_chunk_status, s);
    default: return launch<uint8_t>(d_comp, comp_bytes, d_blk_off, d_col_len, n_chunks, chunk_bytes, ru, d_out, out_bytes, d_chunk_status, s);
  }
}
