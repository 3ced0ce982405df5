// One CTA per RLE chunk: a walk warp finds the headers, the other warps expand them.
//
// A warp that walks the headers of its chunk and expands them one after another leaves 31 lanes idle
// while it reads a header, and a chunk of 128 KiB takes it 0.2 to 0.6 ms whatever the GPU has to
// spare.  Here the two jobs run side by side: in every step the walk warp lists the next headers
// (where each starts, and which value its first is) while the expand warps take the headers of the
// step before, one warp per header, straight from a shared ring of the stream to the output.
//
// More warps run ahead of the walk so that its step from header to header is a look-up or two.  RLE v1
// headers do not say how long they are: a literal group ends with the last of its varints.  So the
// look-ahead writes down, for every byte that ends a varint, where it is (`term`, by ordinal) and how
// many come before each 32 bytes of the stream; each literal's place is a look-up, too.  RLE v2
// headers do say, in a way that takes some 60 instructions to read: the look-ahead reads every byte of
// the stream as if it were a header, 32 at a time, and writes down bytes and values.
//
// Whatever these stages do not expect (a header that does not fit, a base of more than 16 bytes, a literal
// that may be longer than kLongestLiteral, a stream that ends early) is left to the one-warp decoder, which
// starts the chunk over and reports the exact error.
//
// One warp per chunk | a team: RLE v1, 8 MiB of 64-bit values 214 us | 43, 256 MiB of 32-bit values
// 577 | 321 (8 warps; 6, 10 or 12 gain nothing); RLE v2, 3 MB of 16-bit values 434 | 160 (16 warps; 24 or
// 32 are slower from 256 chunks on).  Alone, a chunk waits for the walk (some 60 cycles a header) and the
// barriers between steps; many keep the issue slots 70% busy, mostly with literals' varints.
#pragma once
#include "decode_rle.cuh"

namespace codag_dev {

using TeamRing = InRing<16>;

// A view of a ring for the warps that do not fill it: everything listed for them is resident.
__device__ __forceinline__ TeamRing resident_view(const TeamRing& r) {
  TeamRing v = r;
  v.ready = 0xffffffffu;
  v.release_at = 0xffffffffu;
  return v;
}

struct __align__(16) TeamItem {
  uint32_t pos;   // header, in ring coordinates
  uint32_t n;     // its first value
  uint32_t ord;   // RLE v1 literals: ordinal of the first one's last byte; runs: kRunItem plus the base's bytes
  uint32_t cnt;   // values
};
constexpr uint32_t kRunItem = 0xffffff00u;

constexpr uint32_t kTeamMinBytes = 256;  // a shorter stream is over before a team's stages are under way
constexpr uint32_t kBlockBytes = 2048;  // the look-ahead's step: two slots of the ring
constexpr uint32_t kBlocks = 4;         // blocks whose look-ahead is kept

// how far the chunk has come: of what the warps say in one step, the highest counts
enum : uint32_t { kTeamGo = 0, kTeamDone = 1, kTeamFallback = 2, kTeamTimeout = 3, kTeamShort = 4 };

// The ring's barriers, which outlive a stream where a CTA takes several
struct TeamBars {
  uint64_t bar[16];
  uint32_t phase;
};

template <uint32_t ITEMS>
struct TeamBatch {
  TeamItem item[ITEMS];
  uint32_t items;
  uint32_t first;  // position of its first header: what the ring has to keep
};

// --- RLE v1 -----------------------------------------------------------------------------------------
constexpr uint32_t kV1Items = 128;
struct TeamV1 {
  static constexpr uint32_t kAhead = 2;
  alignas(128) uint8_t ring[TeamRing::kAlloc];
  uint16_t term[kBlocks * kBlockBytes];                  // low half of the position, by ordinal
  uint2 ends[kBlocks * kBlockBytes / 32];                // of 32 bytes: the varint ends, and the ordinal of the first
  TeamBatch<kV1Items> batch[2];
  uint32_t count[kAhead];   // varint ends of the look-ahead warps' slots
  uint32_t prepared, ords;  // blocks done, and varint ends in them
  uint32_t state;
};
constexpr uint32_t kTermMask = kBlocks * kBlockBytes - 1u, kWordMask = kBlocks * kBlockBytes / 32u - 1u;

// Look-ahead warps (me 0 and 1): slot 2 * block + me, 32 bytes a lane, the ordinals going on from `base`.
__device__ __forceinline__ void find_ends(const TeamRing& in, TeamV1& sm, uint32_t block, uint32_t base, uint32_t me,
                                          uint32_t lane) {
  const uint32_t p = block * kBlockBytes + me * kSlotBytes + 32u * lane;
  uint32_t ends = 0;  // bit i: byte p + i ends a varint
#pragma unroll
  for (uint32_t h = 0; h < 2; h++) {
    const uint4 v = ld_s128(in.sbuf + ((p + 16u * h) & TeamRing::kMask));
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (uint32_t k = 0; k < 4; k++)  // the four top bits gathered by a product
      ends |= (((((~w[k] & 0x80808080u) >> 7) * 0x01020408u) >> 24) & 15u) << (16u * h + 4u * k);
  }
  if (p + 32u > in.hi) ends &= p >= in.hi ? 0u : (1u << (in.hi - p)) - 1u;
  if (p < in.lo) ends &= FULL << (in.lo - p);  // lo is below 16
  // A varint of more than kLongestLiteral bytes leaves three of these words in a row without an end, two of them in
  // one slot.  (A look at every literal's length as it is expanded took 6%.)
  static_assert(kLongestLiteral >= 127);
  const uint32_t none = __ballot_sync(FULL, !ends && p + 32u <= in.hi);
  if ((none & (none >> 1)) && lane == 0) atomicMax(&sm.state, static_cast<uint32_t>(kTeamFallback));
  uint32_t upto = __popc(ends);
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t o = __shfl_up_sync(FULL, upto, d);
    if (lane >= static_cast<uint32_t>(d)) upto += o;
  }
  if (lane == 31) sm.count[me] = upto;
  asm volatile("bar.sync 1, 64;" ::: "memory");
  if (me) base += sm.count[0];
  base += upto - __popc(ends);
  sm.ends[(p >> 5) & kWordMask] = make_uint2(ends, base);
  for (uint32_t m = ends; m; m &= m - 1u) sm.term[base++ & kTermMask] = static_cast<uint16_t>(p + __ffs(m) - 1u);
}

// Walk warp, one lane: headers from `pos` (value n) into `b` while their ends are known.
__device__ __forceinline__ void walk_v1(const TeamRing& in, TeamV1& sm, TeamBatch<kV1Items>& b, uint32_t& pos, uint32_t& n,
                                        uint32_t cap, uint32_t blocks, bool stuck) {
  const uint32_t ords = sm.ords, known = sm.prepared * kBlockBytes;
  const bool all = sm.prepared >= blocks;
  const uint32_t limit = all ? in.hi : known;
  uint32_t items = 0, state = kTeamGo;
  b.first = pos;
  while (items < kV1Items) {
    if (n >= cap) {
      state = kTeamDone;
      break;
    }
    if (pos + 2u >= limit) {
      if (!all) break;
      // a literal group of one one-byte value may end the stream, a run may not
      if (pos + 2u > limit || in.rd8(pos) < 0x80u) {
        state = kTeamFallback;
        break;
      }
    }
    const uint32_t h = in.rd8(pos), a = pos + 1u;
    const uint2 e = sm.ends[(a >> 5) & kWordMask];
    const uint32_t rank = e.y + __popc(e.x & ((1u << (a & 31u)) - 1u));  // ordinal of the first varint end from a on
    const bool run = h < 0x80u;  // run: the base's varint starts a byte later, and that byte may be an end, too
    const uint32_t cnt = run ? h + 3u : 256u - h;
    const uint32_t last = rank + (run ? (e.x >> (a & 31u)) & 1u : cnt - 1u);
    const uint32_t q = run ? a + 1u : a;
    const uint32_t bytes = ((sm.term[last & kTermMask] - q) & 0xffffu) + 1u;
    if (last >= ords || n + cnt > cap || (run && bytes > 16u)) {
      if (last < ords || all) state = kTeamFallback;
      break;
    }
    b.item[items++] = TeamItem{pos, n, run ? kRunItem + bytes : rank, cnt};
    pos = q + bytes;
    n += cnt;
  }
  if (stuck && items == 0 && state == kTeamGo) state = kTeamFallback;  // longer than the look-ahead
  b.items = items;
  if (state != kTeamGo) atomicMax(&sm.state, state);
}

template <int E>
__device__ __forceinline__ void expand_v1(TeamRing& in, const TeamV1& sm, DirectOut& out, const TeamItem& it, uint32_t lane) {
  constexpr uint64_t M = emask<E>();
  if (it.ord > kRunItem) {
    const int64_t delta = static_cast<int8_t>(in.rd8(it.pos + 1u));
    const uint32_t len = it.ord - kRunItem;
    const uint64_t base = len <= 4u ? leb_compact32(in.peek_le32(it.pos + 2u), len)
                                    : leb_value(in.peek_le64(it.pos + 2u), in.peek_le64(it.pos + 10u), len);
    body_fill<E>(out, it.n, it.cnt, base, static_cast<uint64_t>(delta), lane);
    return;
  }
  for (uint32_t i = lane; i < it.cnt; i += 32) {
    const uint32_t t1 = sm.term[(it.ord + i) & kTermMask];
    const uint32_t t0 = i ? sm.term[(it.ord + i - 1u) & kTermMask] + 1u : it.pos + 1u;
    const uint32_t start = it.pos + ((t0 - it.pos) & 0xffffu), len = ((t1 - t0) & 0xffffu) + 1u;
    uint64_t v;
    if (len <= 4u) {
      v = leb_compact32(in.peek_le32(start), len);
    } else {
      const uint64_t lo8 = in.peek_le64(start);
      v = leb_value(lo8, len > 8u ? in.peek_le64(start + 8u) : 0ull, len);
    }
    put_elem<E>(out, it.n + i, v & M);
  }
}

// --- RLE v2 -----------------------------------------------------------------------------------------
constexpr uint32_t kV2Items = 64;
template <uint32_t AHEAD>
struct TeamV2 {
  static constexpr uint32_t kAhead = AHEAD;
  alignas(128) uint8_t ring[TeamRing::kAlloc];
  uint32_t info[kBlocks * kBlockBytes];  // of a header that starts here: bytes (12 bits), values; 0: not a usual one
  TeamBatch<kV2Items> batch[2];
  uint32_t prepared, ords;  // blocks done
  uint32_t state;
};

// Look-ahead warps: every byte of `block` read as a header (as rlev2_size does for one).
template <uint32_t AHEAD>
__device__ __forceinline__ void read_headers(const TeamRing& in, TeamV2<AHEAD>& sm, uint32_t block, uint32_t me, uint32_t lane) {
#pragma unroll 2
  for (uint32_t g = me; g < kBlockBytes / 32u; g += AHEAD) {
    const uint32_t p = block * kBlockBytes + 32u * g + lane;
    const uint32_t w = in.peek_be32(p);
    // varint ends of the bytes from p + 2 on
    const uint32_t e0 = __ballot_sync(FULL, !(w >> 31) && p < in.hi);
    const uint32_t e1 = __ballot_sync(FULL, in.rd8(p + 32u) < 0x80u && p + 32u < in.hi);
    const uint32_t ends = static_cast<uint32_t>(((static_cast<uint64_t>(e1) << 32) | e0) >> (lane + 2u)) & 0xffu;
    const uint32_t two = ends & (ends - 1u);  // from the second on
    const uint32_t first = w >> 24, kind = w >> 30, enc = (first >> 1) & 0x1fu;
    const uint32_t len8 = (((w >> 16) & 0x1ffu) + 1u) & 0xffu, nd = (len8 - 2u) & 0xffu;
    const uint32_t fbw = v2_width(enc), body = (len8 * fbw + 7u) / 8u;
    uint32_t size, cnt = len8;
    if (kind == 0) {
      size = 2u + ((first >> 3) & 7u);
      cnt = (first & 7u) + 3u;
    } else if (kind == 1) {
      size = 2u + body;
    } else if (kind == 3) {
      size = two ? 2u + __ffs(two) + (enc ? (nd * fbw + 7u) / 8u : 0u) : 0u;
      cnt = nd + 2u;
    } else {
      const uint32_t third = (w >> 8) & 0xffu, fourth = w & 0xffu;
      const uint32_t both = v2_width(third & 0x1fu) + ((fourth >> 5) & 7u) + 1u;
      size = both > 64u ? 0u : 5u + ((third >> 5) & 7u) + body + ((fourth & 0x1fu) * v2_closest(both) + 7u) / 8u;
    }
    sm.info[p & (kBlocks * kBlockBytes - 1u)] = size ? size | (cnt << 12) : 0u;
  }
}

// The same for a DELTA header whose varints take more than 8 bytes, up to 16 each; 0: neither is it that.
static __device__ __noinline__ uint32_t long_delta(const TeamRing& in, uint32_t p) {
  const uint32_t w = in.peek_be32(p);
  if (w >> 30 != 3u) return 0;
  const uint32_t l1 = leb_len(in.peek_le64(p + 2u), in.peek_le64(p + 10u));
  const uint32_t l2 = l1 ? leb_len(in.peek_le64(p + 2u + l1), in.peek_le64(p + 10u + l1)) : 0u;
  if (!l2) return 0;
  const uint32_t enc = (w >> 25) & 0x1fu, nd = (((w >> 16) & 0x1ffu) - 1u) & 0xffu;
  return (2u + l1 + l2 + (enc ? (nd * v2_width(enc) + 7u) / 8u : 0u)) | ((nd + 2u) << 12);
}

// Walk warp, one lane: headers from `pos` (value n) into `b` while they are known.
template <uint32_t AHEAD>
__device__ __forceinline__ void walk_v2(const TeamRing& in, TeamV2<AHEAD>& sm, TeamBatch<kV2Items>& b, uint32_t& pos, uint32_t& n,
                                        uint32_t cap, uint32_t blocks) {
  const bool all = sm.prepared >= blocks;
  const uint32_t known = all ? in.hi : sm.prepared * kBlockBytes;
  uint32_t items = 0, state = kTeamGo;
  b.first = pos;
  while (items < kV2Items) {
    if (pos >= in.hi) {
      state = kTeamDone;
      break;
    }
    if (pos >= known) break;
    uint32_t v = sm.info[pos & (kBlocks * kBlockBytes - 1u)];
    if (!v) {
      if (!all && pos + 64u > known) break;
      v = long_delta(in, pos);
    }
    const uint32_t next = pos + (v & 0xfffu), cnt = v >> 12;
    if (!v || next > in.hi || n + cnt > cap) {
      state = kTeamFallback;
      break;
    }
    if (next > known) break;  // its bytes are not all there yet
    b.item[items++] = TeamItem{pos, n, 0, cnt};
    pos = next;
    n += cnt;
  }
  b.items = items;
  if (state != kTeamGo) atomicMax(&sm.state, state);
}

// Whether one warp decodes an RLE v2 stream faster.  A team reads every byte as a header, 2.1 us per KiB; a warp
// expands DIRECT groups in some 3 us per 1024 values and 0.6 per KiB, but takes longer over other headers.  So
// streams of more than two bytes a value that begin with DIRECT groups are left to a warp (128 KiB of random 64-bit
// values: 284 us by a team | 138, of 32-bit values 286 | 186, of 16-bit values, 2.02 bytes each, 343 | 292).
// (Finding out in the walk, header by header, made it 5 to 17% slower for all.)
__device__ __forceinline__ bool rlev2_alone(const uint8_t* src, uint32_t len, uint32_t values) {
  if (len <= 2ull * values) return false;
  uint32_t p = 0;
  for (uint32_t h = 0; h < 8 && p + 2u <= len; h++) {
    const uint32_t first = __ldg(src + p), len8 = ((((first & 1u) << 8) | __ldg(src + p + 1u)) + 1u) & 0xffu;
    if (first >> 6 != 1u) return false;
    p += 2u + (len8 * v2_width((first >> 1) & 0x1fu) + 7u) / 8u;
  }
  return true;
}

// The stream src[0, len) by all WARPS warps of the CTA: warp 0 walks, the next kAhead look ahead (the
// first of them fills the ring), the others expand.  kTeamDone, kTeamShort when the stream ends before
// `store` bytes, kTeamTimeout, or kTeamFallback: the one-warp decoder has to start it over.
template <int CODEC, int E, uint32_t WARPS, class Team>
__device__ __forceinline__ uint32_t rle_team(Team& sm, TeamBars& tb, const uint8_t* src, uint32_t len, uint8_t* dst,
                                             uint32_t store, uint32_t cap, uint64_t wait_cycles) {
  constexpr bool V1 = CODEC == CODAG_CODEC_RLEV1;
  constexpr uint32_t kFirst = 1u + Team::kAhead, kExpand = WARPS - kFirst;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  TeamRing in;
  in.buf = sm.ring;
  in.sbuf = smem_u32(sm.ring);
  in.bar = tb.bar;
  in.phase = tb.phase;
  in.wait_cycles = wait_cycles;
  in.lane = lane;
  in.begin(src, len);
  if (threadIdx.x == 0) {
    sm.state = kTeamGo;
    sm.batch[0].items = sm.batch[1].items = 0;
    sm.batch[0].first = sm.batch[1].first = in.lo;
    sm.prepared = sm.ords = 0;
  }
  __syncthreads();
  DirectOut o;
  o.lane = lane;
  o.begin(dst, store);
  uint32_t pos = in.lo, n = 0;  // the walk
  uint32_t prepared = 0;        // blocks looked over so far
  uint32_t state;
  const uint32_t blocks = (in.hi + kBlockBytes - 1u) / kBlockBytes;
  for (uint32_t k = 0;; k ^= 1u) {  // the walk fills batch k while batch k ^ 1 is expanded
    auto& mine = sm.batch[k];
    const auto& prev = sm.batch[k ^ 1u];
    const uint32_t keep = prev.first;  // what comes before it is done with
    const bool room = prepared < keep / kBlockBytes + kBlocks, ahead = prepared < blocks && room;
    if (warp == 0) {
      if (lane == 0) {
        if constexpr (V1) walk_v1(in, sm, mine, pos, n, cap, blocks, prev.items == 0 && !room);
        else walk_v2(in, sm, mine, pos, n, cap, blocks);
      }
      __syncwarp();
    } else if (warp < kFirst) {
      if (ahead) {
        if (warp == 1) {  // RLE v2 headers are read from some bytes past the block, too
          const uint32_t end = (prepared + 1u) * kBlockBytes + (V1 ? 0u : 64u);
          if ((!in.release(keep) || in.ensure(end < in.hi ? end : in.hi)) && lane == 0)
            atomicMax(&sm.state, static_cast<uint32_t>(kTeamTimeout));
        }
        asm volatile("bar.sync 1, %0;" ::"n"(32 * Team::kAhead) : "memory");
        if constexpr (V1) find_ends(in, sm, prepared, sm.ords, warp - 1u, lane);
        else read_headers(in, sm, prepared, warp - 1u, lane);
      }
    } else {
      TeamRing view = resident_view(in);
      for (uint32_t i = warp - kFirst; i < prev.items; i += kExpand) {
        const TeamItem it = prev.item[i];
        if constexpr (V1) {
          expand_v1<E>(view, sm, o, it, lane);
        } else {
          uint32_t p = it.pos, v = it.n;
          if (rlev2_header<16, E>(view, o, p, v, cap, in.hi, lane) && lane == 0)
            atomicMax(&sm.state, static_cast<uint32_t>(kTeamFallback));
        }
      }
    }
    __syncthreads();
    state = sm.state;
    const bool last = mine.items == 0;
    __syncthreads();  // everyone has seen this step's state before the next one changes it
    if (ahead) {
      prepared++;
      if (threadIdx.x == 0) {
        sm.prepared = prepared;
        if constexpr (V1) sm.ords += sm.count[0] + sm.count[1];
      }
    }
    __syncthreads();
    if (state >= kTeamFallback || (state == kTeamDone && last)) break;
  }
  if (warp == 1) {
    if (!in.drain()) state = kTeamTimeout;
    if (lane == 0) {
      sm.batch[0].items = state;
      tb.phase = in.phase;  // the next stream through this ring goes on from here
    }
  }
  if (warp == 0 && lane == 0) sm.batch[0].first = n;
  __syncthreads();
  state = sm.batch[0].items;
  return state == kTeamDone && static_cast<uint64_t>(sm.batch[0].first) * E < o.store ? kTeamShort : state;
}

}  // namespace codag_dev
