// One warp for a whole Deflate (RFC 1951) chunk, for chunks that are not worth a team of six
// (decode_deflate.cuh): where there are many and they are small, or nearly all stored blocks or long runs.
//
// Every lane runs the same symbol loop on the same data (shared-memory reads broadcast), so only the stores
// differ from lane to lane: some 140 warp instructions a symbol, but nothing to hand over, and seven times as many
// chunks on the GPU at once.  Output goes through a window in shared memory; sources further back are read
// from the chunk's output.  A team's part of an SM is busy 35 us with the smallest chunk (tables, barriers):
// 65536 chunks of 1 KiB of text 6130 us by teams | 2810 by warps, 16384 of 4 KiB of zeros 1419 | 204, of random bytes
// 214 | 73; but one chunk of 16 KiB of text 115 | 1400.  32 warps a SM with windows of 1 KiB are faster than 22 with
// 4 KiB (4 KiB chunks of text 2433 us | 2624), and more registers for fewer warps are no gain either.
#pragma once
#include "decode_deflate.cuh"

namespace codag_dev {

constexpr uint32_t kWarpLitLB = 9, kWarpDistLB = 7;  // the distance table also holds the code-length codes
static_assert(kWarpDistLB == kCodeLenLB);

using InflateWarpWin = OutRing<10, 8>;

// One warp's tables.
struct InflateWarp {
  uint32_t lit_lut[1u << kWarpLitLB];
  uint32_t dist_lut[1u << kWarpDistLB];
  uint32_t lit_cnt[16], lit_first[16], lit_index[16];
  uint32_t dist_cnt[16], dist_first[16], dist_index[16];
  uint32_t fill[16];
  uint16_t lit_sorted[288];
  uint16_t dist_sorted[32];
  uint8_t lens[320];
  __device__ __forceinline__ HuffTable lit() { return {lit_lut, lit_sorted, lit_cnt, lit_first, lit_index}; }
  __device__ __forceinline__ HuffTable dist() { return {dist_lut, dist_sorted, dist_cnt, dist_first, dist_index}; }
};

// The stream's next bits, refilled a word at a time.
template <int NSLOT>
struct BitReader {
  uint64_t bb;    // pending bits, the next in bit 0
  uint32_t bc;    // how many
  uint32_t wpos;  // ring position of the next word (a multiple of 4)

  __device__ __forceinline__ int refill(InRing<NSLOT>& in) {
    if (wpos < in.hi) {
      const uint32_t end = min(wpos + 4u, in.hi);
      if (end > in.ready) {
        // a stored block's first bytes may be in the buffer
        if (!in.release(wpos >= 8u ? wpos - 8u : 0u)) return CODAG_ETIMEOUT;
        const int st = in.ensure(end);
        if (st) return st;
      }
    } else if (wpos > in.hi + 16u) {
      return CODAG_ECORRUPT;
    }
    bb |= static_cast<uint64_t>(in.rd32(wpos)) << bc;
    bc += 32;
    wpos += 4;
    return CODAG_OK;
  }
  // goes on at byte p
  __device__ __forceinline__ int start(InRing<NSLOT>& in, uint32_t p) {
    wpos = p & ~3u;
    bb = 0;
    bc = 0;
    const int st = refill(in);
    if (!st) drop(8u * (p & 3u));
    return st;
  }
  __device__ __forceinline__ void drop(uint32_t n) {
    bb >>= n;
    bc -= n;
  }
  __device__ __forceinline__ uint32_t low() const { return static_cast<uint32_t>(bb); }
  __device__ __forceinline__ uint64_t pos() const { return static_cast<uint64_t>(wpos) * 8u - bc; }  // of the next bit
};

template <int NSLOT, class OUT>
struct WarpInflater {
  InRing<NSLOT>& in;
  OUT& out;
  InflateWarp& sc;
  uint32_t cap, lane;
  uint32_t op;  // bytes written
  BitReader<NSLOT> br;

  __device__ __forceinline__ int at_least(uint32_t bits) { return br.bc < bits ? br.refill(in) : static_cast<int>(CODAG_OK); }

  __device__ __forceinline__ int stored() {
    br.drop(br.bc & 7u);
    int st = at_least(32);
    if (st) return st;
    const uint32_t len = br.low() & 0xffffu;
    if (len != (~(br.low() >> 16) & 0xffffu)) return CODAG_ECORRUPT;
    br.drop(32);
    uint32_t p = br.wpos - br.bc / 8u;
    if (p + len > in.hi || op + len > cap) return CODAG_ECORRUPT;
    constexpr uint32_t kPiece = (NSLOT - 1) * kSlotBytes < OUT::kBytes - OUT::kFlush ? (NSLOT - 1) * kSlotBytes
                                                                                    : OUT::kBytes - OUT::kFlush;
    for (uint32_t left = len; left;) {
      const uint32_t piece = left < kPiece ? left : kPiece;
      if (!in.release(p)) return CODAG_ETIMEOUT;
      st = in.ensure(p + piece);
      if (st) return st;
      for (uint32_t t = lane; t < piece; t += 32) out.put8(op + t, in.rd8(p + t));
      op += piece;
      p += piece;
      left -= piece;
      __syncwarp();
      out.flush_to(op);
    }
    return br.start(in, p);
  }

  __device__ __forceinline__ bool tables(uint32_t hlit, const uint8_t* dlens, uint32_t hdist) {
    __syncwarp();
    if (!order_codes(sc.lens, hlit, sc.lit(), sc.fill, lane)) return false;
    if (!order_codes(dlens, hdist, sc.dist(), sc.fill, lane)) return false;
    __syncwarp();
    fill_table<kWarpLitLB, kAlphaLitLen>(sc.lit(), lane, 32);
    fill_table<kWarpDistLB, kAlphaDist>(sc.dist(), lane, 32);
    __syncwarp();
    pair_literals<kWarpLitLB>(sc.lit_lut, lane, 32);
    __syncwarp();
    return true;
  }

  __device__ __forceinline__ int fixed() {  // RFC 1951 3.2.6
    __syncwarp();
    for (uint32_t s = lane; s < 320; s += 32) sc.lens[s] = s < 144 ? 8 : s < 256 ? 9 : s < 280 ? 7 : s < 288 ? 8 : 5;
    return tables(288, sc.lens + 288, 30) ? CODAG_OK : CODAG_ECORRUPT;
  }

  __device__ __forceinline__ int dynamic() {  // zlib.h:607-707
    int st = at_least(32);
    if (st) return st;
    const uint32_t hlit = (br.low() & 31u) + 257u, hdist = ((br.low() >> 5) & 31u) + 1u, hclen = ((br.low() >> 10) & 15u) + 4u;
    br.drop(14);
    if (hlit > 286 || hdist > 30) return CODAG_ECORRUPT;
    __syncwarp();
    for (uint32_t i0 = 0; i0 < 19; i0 += 10) {  // code length code lengths, ten at a time
      st = at_least(32);
      if (st) return st;
      const uint32_t i = i0 + lane;
      if (lane < 10 && i < 19) sc.lens[kCodeLenOrder[i]] = i < hclen ? static_cast<uint8_t>((br.low() >> (3u * lane)) & 7u) : 0;
      br.drop(3u * (hclen > i0 ? min(hclen - i0, 10u) : 0u));
    }
    __syncwarp();
    if (!order_codes(sc.lens, 19, sc.dist(), sc.fill, lane)) return CODAG_ECORRUPT;
    __syncwarp();
    fill_table<kCodeLenLB, kAlphaCodeLen>(sc.dist(), lane, 32);
    __syncwarp();
    const uint32_t s_cl = smem_u32(sc.dist_lut), total = hlit + hdist;
    uint32_t idx = 0, prev = 0;
    while (idx < total) {  // run-length coded with symbols 16..18
      st = at_least(32);
      if (st) return st;
      const uint32_t e = ld_s32(s_cl + 4u * (br.low() & ((1u << kCodeLenLB) - 1u)));
      if (e & kSlowFlag) return CODAG_ECORRUPT;  // code lengths are at most 7 bits
      br.drop(e & 31u);
      const uint32_t sym = e >> 16;
      uint32_t rep = 1, val = sym;
      if (sym >= 16) {
        if (sym == 16 && idx == 0) return CODAG_ECORRUPT;
        const uint32_t bits = sym == 16 ? 2u : sym == 17 ? 3u : 7u;
        val = sym == 16 ? prev : 0u;
        rep = (sym == 18 ? 11u : 3u) + (br.low() & ((1u << bits) - 1u));
        br.drop(bits);
        if (idx + rep > total) return CODAG_ECORRUPT;
      }
      for (uint32_t t = lane; t < rep; t += 32) sc.lens[idx + t] = static_cast<uint8_t>(val);
      prev = val;
      idx += rep;
    }
    __syncwarp();
    if (sc.lens[256] == 0) return CODAG_ECORRUPT;
    return tables(hlit, sc.lens + hlit, hdist) ? CODAG_OK : CODAG_ECORRUPT;
  }

  // len bytes from `dist` before op
  __device__ __forceinline__ void match(uint32_t len, uint32_t dist) {
    const uint32_t src = op - dist;
    uint32_t r = dist >= len ? lane : lane % dist;
    const uint32_t step = dist >= len ? 32u : 32u % dist;
    __syncwarp();  // the window's last bytes
    if (dist + len <= OUT::kBytes) {
      for (uint32_t t = lane; t < len; t += 32) {
        out.put8(op + t, out.get8(src + r));
        r += step;
        if (dist < len && r >= dist) r -= dist;
      }
    } else {  // further back: these bytes were flushed (what is not stored is not needed either)
      for (uint32_t t = lane; t < len; t += 32) {
        const uint32_t p = src + r;
        out.put8(op + t, p < out.store ? out.gdst[p] : 0u);
        r += step;
        if (dist < len && r >= dist) r -= dist;
      }
    }
    __syncwarp();
  }

  __device__ __forceinline__ int symbols() {  // zlib.h:712-805
    const uint32_t s_lit = smem_u32(sc.lit_lut), s_dist = smem_u32(sc.dist_lut);
    const uint32_t lit_sh = 16u + 8u * (lane & 1u);  // the first literal in bits 16-23, the second in 24-31
    for (;;) {
      int st = at_least(32);
      if (st) return st;
      uint32_t e = ld_s32(s_lit + 4u * (br.low() & ((1u << kWarpLitLB) - 1u)));
      if (e & kSlowFlag) e = slow_entry<kWarpLitLB>(br.low(), sc.lit(), kAlphaLitLen);
      const uint32_t lo = br.low();
      br.drop(e & 31u);
      if ((e & kKindMask) == kKindLitBits) {  // one literal or two, by the first lanes
        const uint32_t pair = (e >> 11) & 1u;
        if (lane <= pair) out.put8(op + lane, e >> lit_sh);
        op += 1u + pair;
      } else if ((e & kKindMask) == kKindLenBits) {
        const uint32_t ln = (e >> 5) & 15u, len = (e >> 16) + bfe32(lo, ln, (e & 31u) - ln);
        st = at_least(28);  // a distance code and its extra bits
        if (st) return st;
        uint32_t d = ld_s32(s_dist + 4u * (br.low() & ((1u << kWarpDistLB) - 1u)));
        if (d & kSlowFlag) d = slow_entry<kWarpDistLB>(br.low(), sc.dist(), kAlphaDist);
        if (d & kKindMask) return CODAG_ECORRUPT;
        const uint32_t dn = (d >> 5) & 15u, dt = d & 31u, dist = (d >> 16) + 1u + bfe32(br.low(), dn, dt - dn);
        br.drop(dt);
        if (dist > op || op + len > cap) return CODAG_ECORRUPT;
        match(len, dist);
        op += len;
      } else {
        return (e & kKindMask) == kKindEndBits ? CODAG_OK : CODAG_ECORRUPT;
      }
      if (op - out.flushed >= OUT::kFlush) {
        if (op > cap) return CODAG_ECORRUPT;
        out.flush_to(op);
      }
    }
  }

  // The stream bound to `in`, `wrapper` header bytes first.
  __device__ __forceinline__ int run(uint32_t wrapper) {
    const uint64_t end = static_cast<uint64_t>(in.hi) * 8u;
    if (in.lo + wrapper > in.hi) return CODAG_ECORRUPT;
    if (!in.release(in.lo)) return CODAG_ETIMEOUT;
    int st = br.start(in, in.lo + wrapper);
    bool last = false, have_fixed = false;
    while (!st && !last) {
      if (br.pos() >= end) return CODAG_ECORRUPT;
      st = at_least(32);
      if (st) return st;
      last = br.low() & 1u;
      const uint32_t btype = (br.low() >> 1) & 3u;
      br.drop(3);
      if (btype == 0) {
        st = stored();
        continue;
      }
      if (btype == 3) return CODAG_ECORRUPT;
      if (btype == 2 || !have_fixed) st = btype == 2 ? dynamic() : fixed();
      have_fixed = btype == 1;
      if (!st) st = symbols();
    }
    return st || br.pos() <= end ? st : static_cast<int>(CODAG_ECORRUPT);
  }
};

// What a chunk takes, in ns: a team's place (three a SM), or one warp, of which 32 a SM take 1.6 times as long; fitted
// to text, columns, zeros and random bytes in chunks of 1 to 128 KiB (64 MiB of each, and few chunks).
struct InflateCost {
  float team, warp;
};
__host__ __device__ __forceinline__ InflateCost inflate_cost(uint64_t out_bytes, uint64_t stream) {
  const float o = static_cast<float>(out_bytes), s = static_cast<float>(stream);
  if (stream >= out_bytes && stream <= out_bytes + out_bytes / 64u + 64u)  // stored blocks
    return {4000.f + 0.6f * o, 4000.f + 1.9f * o};
  return {34000.f + 1.5f * o + 14.f * s, 15000.f + 3.1f * o + 270.f * s};
}

// The chunk's status; `in` is bound to its stream, `out` to its output.
template <int NSLOT, class OUT>
__device__ __forceinline__ int inflate_warp(InRing<NSLOT>& in, OUT& out, InflateWarp& sc, uint64_t chunk_bytes, uint32_t wrapper,
                                            uint32_t lane) {
  WarpInflater<NSLOT, OUT> d{in, out, sc, static_cast<uint32_t>(chunk_bytes), lane, 0, {}};
  int st = d.run(wrapper);
  if (!in.drain() && !st) st = CODAG_ETIMEOUT;
  out.finish(d.op);
  return st || (d.op >= out.store && d.op <= d.cap) ? st : static_cast<int>(CODAG_ECORRUPT);
}

}  // namespace codag_dev
