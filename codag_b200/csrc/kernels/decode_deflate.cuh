// Team decoder for one Deflate (RFC 1951) chunk: six warps in four stages.
//
// CODAG's decoder (include/zlib/zlib.h:807-902) runs one symbol at a time on all 32 lanes
// of a warp.  So did the first kernels here, and they spent about 140 warp instructions on every
// symbol.  This decoder puts the lanes to work on different symbols:
//
//   - Scan (two warps, 64 lanes).  A Huffman bit stream read from a wrong bit falls into step with
//     the right symbol boundaries after a while (text compressed by zlib at level 6: after 106 bits
//     on average, in 99% of the cases within 512).  The lanes cut the next stretch of a block into
//     64 pieces.  Each warms up kWarmBits before its piece to guess where the piece's first symbol
//     starts, decodes the piece from there, and notes where every kCell-th symbol begins.  A lane
//     whose start turns out not to be the end of the lane below decodes once more, until the chain
//     from lane 0, whose start is known, holds.  So the result is the serial decoder's, whatever
//     the guesses were.
//   - Tokens (two warps, taking turns).  Decodes the noted cells again, 32 at a time, this time from
//     known starts, into a dense list of tokens, and marks the byte each token starts at in a bit
//     map.  Decoding twice is cheaper than keeping every lane's tokens: their number varies too much
//     from piece to piece to give each lane room of its own.
//   - Place (one warp).  Finds the token that covers each output byte by counting the marks up to it,
//     32 bytes per step and eight steps side by side.
//   - Copy (one warp).  Takes each byte's literal, or the byte `distance` before it from a 32 KiB
//     shared-memory window (the largest distance Deflate has, so no source is ever read back from
//     global memory).  A source inside the same 32 bytes is followed lane to lane.
//
// Stored blocks pass the stages in between by: the copy warp takes their bytes from the stream, and the
// input rings go on behind them (128 KiB of stored blocks: 226 us as tokens, 71 now; 512 chunks 461 | 154).  So do
// long matches that follow one another at one distance, as in runs of a byte or of a record: the copy warp
// repeats it over all of them (128 KiB of zeros: 602 us byte by byte, 147 now).
//
// The stages run as a pipeline, handing over in buffers guarded by named barriers, so no warp spins.
// Each stage is one or two warps' chain of dependent instructions, about six cycles each, which is
// why the work is spread over as many warps as it is.
//
// Text in 128 KiB chunks (zlib level 6), one symbol at a time on one or two warps | by teams:
// 256 MiB 8.6 ms | 2.3, 8 MiB 6.8 ms | 0.40, 200 KB 6.6 ms | 0.39; a 40 MB column in 64 KiB chunks of
// level 9 6.3 ms | 0.84.  (Many small chunks are left to single warps, decode_deflate_warp.cuh.)  A lone chunk takes 0.37 ms: the scan's chain of table look-ups, some 310 cycles
// a symbol for 64 lanes (warm-up 30%, pieces 45%, headers and tables 9%).  With three teams on every SM
// all stages slow down together, a third of the issue slots used and a third of the stalls waiting for
// instructions: seven different loops compete for the instruction cache, so what makes them longer
// (unrolling, predication instead of branches) loses there what it gains alone.
#pragma once
#include "device_common.cuh"

namespace codag_dev {

// Length code k = symbol - 257 and distance code k (RFC 1951 3.2.5), computed: 32 lanes at different
// codes would read a table in constant memory one after another.
__device__ __forceinline__ uint32_t len_extra(uint32_t k) { return k < 8 || k == 28 ? 0u : (k >> 2) - 1u; }
__device__ __forceinline__ uint32_t len_base(uint32_t k) {
  return k < 8 ? k + 3u : k == 28 ? 258u : ((4u + (k & 3u)) << ((k >> 2) - 1u)) + 3u;
}
__device__ __forceinline__ uint32_t dist_extra(uint32_t k) { return k < 4 ? 0u : (k >> 1) - 1u; }
__device__ __forceinline__ uint32_t dist_base(uint32_t k) { return k < 4 ? k + 1u : ((2u + (k & 1u)) << ((k >> 1) - 1u)) + 1u; }
__constant__ uint8_t kCodeLenOrder[19] = {16, 17, 18, 0, 8, 7, 9, 6, 10, 5, 11, 4, 12, 3, 13, 2, 14, 1, 15};

constexpr uint32_t kLitLB = 10;  // codes of 11 and more bits: 0.02-0.3% of the symbols measured
constexpr uint32_t kDistLB = 8;   // of 9 and more bits: 0.2-0.8% of the distances
constexpr uint32_t kCodeLenLB = 7;

// Table entry (32 bits):
//   [0,5)   bits consumed in all: code length + extra bits, or both codes of a literal pair
//   [5,9)   code length of the (first) symbol
//   [9,11)  kind: literal, length, end of block, other (invalid, or not in the table)
//   [11]    a second literal follows in [24,32) (literal/length tables only)
//   [12]    the code is longer than the table: decode it with slow_entry
//   [16,32) literal byte in [16,24) / length base / distance base less one / code-length symbol
enum : uint32_t {
  kKindShift = 9,
  kKindMask = 3u << kKindShift,
  kKindLitBits = 0u,
  kKindLenBits = 1u << kKindShift,
  kKindEndBits = 2u << kKindShift,
  kKindBadBits = 3u << kKindShift,
  kPairFlag = 1u << 11,
  kSlowFlag = 1u << 12,
  kSlowEntry = kKindBadBits | kSlowFlag,
};
enum : int { kAlphaLitLen = 0, kAlphaDist = 1, kAlphaCodeLen = 2 };

__device__ __forceinline__ uint32_t entry_bits(uint32_t total, uint32_t len) { return total | (len << 5); }

__device__ __forceinline__ uint32_t make_entry(uint32_t sym, uint32_t len, int alpha) {
  if (alpha == kAlphaLitLen) {
    if (sym < 256) return entry_bits(len, len) | kKindLitBits | (sym << 16);
    if (sym == 256) return entry_bits(len, len) | kKindEndBits;
    if (sym <= 285) {
      const uint32_t k = sym - 257;
      return entry_bits(len + len_extra(k), len) | kKindLenBits | (len_base(k) << 16);
    }
    return entry_bits(len, len) | kKindBadBits;
  }
  if (alpha == kAlphaDist) {
    if (sym < 30) return entry_bits(len + dist_extra(sym), len) | ((dist_base(sym) - 1u) << 16);
    return entry_bits(len, len) | kKindBadBits;
  }
  return entry_bits(len, len) | (sym << 16);
}

// `n` bits of `x` starting at bit `pos` (pos + n <= 32; n may be 0)
__device__ __forceinline__ uint32_t bfe32(uint32_t x, uint32_t pos, uint32_t n) {
  uint32_t r;
  asm("bfe.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(x), "r"(pos), "r"(n));
  return r;
}

struct HuffTable {
  uint32_t* lut;     // 1 << LB entries
  uint16_t* sorted;  // symbols ordered by (code length, symbol)
  uint32_t* cnt;     // [16] codes per length
  uint32_t* first;   // [16] first canonical code per length
  uint32_t* index;   // [16] position of the first code of each length in `sorted`
};

// Orders the codes of lens[0..nsym) into `t`, without its look-up table.  False when the lengths
// over-subscribe the code space.  Incomplete codes are accepted; their unused codes decode as invalid.
static __device__ __noinline__ bool order_codes(const uint8_t* lens, uint32_t nsym, HuffTable t, uint32_t* fill, uint32_t lane) {
  if (lane < 16) t.cnt[lane] = 0;
  __syncwarp();
  for (uint32_t s = lane; s < nsym; s += 32) {
    const uint32_t l = lens[s];
    if (l) atomicAdd(&t.cnt[l], 1u);
  }
  __syncwarp();
  uint32_t ok = 1;
  if (lane == 0) {
    uint32_t code = 0, idx = 0;
    int left = 1;
    for (uint32_t l = 1; l < 16; l++) {
      t.first[l] = code;
      code = (code + t.cnt[l]) << 1;
      t.index[l] = idx;
      fill[l] = idx;
      idx += t.cnt[l];
      left = (left << 1) - static_cast<int>(t.cnt[l]);
      if (left < 0) ok = 0;
    }
  }
  ok = __shfl_sync(FULL, ok, 0);
  __syncwarp();
  if (!ok) return false;
  for (uint32_t s0 = 0; s0 < nsym; s0 += 32) {
    const uint32_t s = s0 + lane;
    const uint32_t l = s < nsym ? lens[s] : 0u;
    const uint32_t grp = __match_any_sync(FULL, l);
    const uint32_t rank = __popc(grp & lanemask_lt(lane));
    if (l) t.sorted[fill[l] + rank] = static_cast<uint16_t>(s);
    __syncwarp();
    if (l && rank == 0) fill[l] += __popc(grp);
    __syncwarp();
  }
  return true;
}

// The look-up table of ordered codes, by `threads` threads of which this is number `id`.  Canonical codes
// tile the code space in MSB-first order, shorter ones first: slot x's code length is one more than the
// number of lengths whose codes all lie below its prefix.
template <uint32_t LB, int ALPHA>
__device__ __noinline__ void fill_table(HuffTable t, uint32_t id, uint32_t threads) {
  uint32_t end[LB];  // where the codes of each length end, as LB-bit prefixes
#pragma unroll
  for (uint32_t l = 1; l <= LB; l++) end[l - 1] = (t.first[l] + t.cnt[l]) << (LB - l);
  for (uint32_t x = id; x < (1u << LB); x += threads) {
    const uint32_t v = __brev(x) >> (32 - LB);  // MSB-first code prefix of table slot x
    uint32_t len = 1;
#pragma unroll
    for (uint32_t l = 1; l <= LB; l++) len += v >= end[l - 1] ? 1u : 0u;
    t.lut[x] = len <= LB ? make_entry(t.sorted[t.index[len] + (v >> (LB - len)) - t.first[len]], len, ALPHA)
                         : static_cast<uint32_t>(kSlowEntry);
  }
}

// Literal pairs: when the bits of slot x after its literal code hold a whole literal code too, the entry
// carries both.  Only the first-literal fields of the other slot are read, and a pair rewrite leaves
// those fields unchanged, so threads need no order.
template <uint32_t LB>
__device__ __forceinline__ void pair_literals(uint32_t* lut, uint32_t id, uint32_t threads) {
  for (uint32_t x = id; x < (1u << LB); x += threads) {
    const uint32_t e1 = lut[x];
    const uint32_t l1 = (e1 >> 5) & 15u;
    const uint32_t e2 = lut[x >> l1];
    const uint32_t l2 = (e2 >> 5) & 15u;
    if (((e1 | e2) & (kKindMask | kSlowFlag)) == kKindLitBits && l1 + l2 <= LB)
      lut[x] = (e1 & ~31u & 0x00ffffffu) | (l1 + l2) | kPairFlag | ((e2 & 0x00ff0000u) << 8);
  }
}

// Codes longer than the table width: the range of lengths LB+1..15 that holds the bits (zlib.h:459-527
// walks 6..15), all looked at side by side.
template <uint32_t LB>
__device__ __forceinline__ uint32_t slow_entry(uint32_t bits, HuffTable t, int alpha) {
  const uint32_t rev = __brev(bits);
  uint32_t len = 0, at = 0;
#pragma unroll
  for (uint32_t l = LB + 1; l < 16; l++) {
    const uint32_t k = (rev >> (32 - l)) - t.first[l];
    if (k < t.cnt[l]) {
      len = l;
      at = t.index[l] + k;
    }
  }
  return len ? make_entry(t.sorted[at], len, alpha) : static_cast<uint32_t>(kKindBadBits);
}

// Tables of one block.
struct InflateTables {
  uint32_t lit_lut[1u << kLitLB];
  uint32_t dist_lut[1u << kDistLB];
  uint32_t lit_cnt[16], lit_first[16], lit_index[16];
  uint32_t dist_cnt[16], dist_first[16], dist_index[16];
  uint16_t lit_sorted[288];
  uint16_t dist_sorted[32];
  __device__ __forceinline__ HuffTable lit() { return {lit_lut, lit_sorted, lit_cnt, lit_first, lit_index}; }
  __device__ __forceinline__ HuffTable dist() { return {dist_lut, dist_sorted, dist_cnt, dist_first, dist_index}; }
};

constexpr uint32_t kPieces = 64;
constexpr uint32_t kCell = 15;         // symbols from one noted start to the next, or one more or less
constexpr uint32_t kCellMax = 16;      // where two literals were read at once
constexpr uint32_t kCells = 13;        // noted starts of one piece: an odd row spreads over the banks
// A piece aims at kPieceTokens symbols (by the last stretch's bits per symbol), so far below the
// kCell * kCells it may hold that few stretches end early at a full row, and is at most kMaxSpan words
// long, so that 64 pieces fit the 7 KiB of the input ring that are resident behind any read position.
// (Longer pieces, in a ring of twice the size, warm up less often but lose more where a block ends in
// the stretch: as many turns on text, a fifth more on columns.)  Spans are odd numbers of words: the
// lanes' first words lie in different banks.  What is left of a short stream is cut into pieces of kMinSpan
// (chunks of 1 KiB of text 416 us, 462 with 13; a chunk of zeros, where 13 words overfill a row, 147 | 170).
constexpr uint32_t kPieceTokens = 90;
constexpr uint32_t kMinSpan = 5, kMaxSpan = 27;
constexpr uint32_t kWarmBits = 640;

enum : uint32_t { kBatchTokens = 0, kBatchStored = 1, kBatchDone = 2 };
struct ScanBatch {
  // bit offset of each cell from its piece's first bit; cell j starts with symbol kCell * j, or the
  // next where bit 15 is set
  uint16_t row[kPieces * kCells];
  uint16_t cnt[kPieces];  // of each piece: symbols in bits 0-7, noted starts above
  uint32_t kind;
  uint32_t base;   // first bit (kBatchTokens), first byte (kBatchStored), in ring coordinates
  uint32_t size;   // bits per piece, or bytes
  uint32_t table;
  int32_t status;  // with kBatchDone
};

// Token: where its bytes come from in the low half (bit 15 set: the literal in bits 0-7; clear: the
// distance less one), how many they are in the high half.
constexpr uint32_t kLiteral = 0x8000u, kLiteralToken = 0x18000u;
constexpr uint32_t kTokens = 32 * kCellMax;
constexpr uint32_t kRange = 3072;  // output bytes of one token batch
struct TokenBatch {
  uint32_t starts[kRange / 32];  // bit b: a token starts at byte b of the range
  uint32_t list;    // which of the token warp's lists
  uint32_t before;  // its tokens that start before the range; kStored: where the bytes are in the
                    // stream; kRepeat: the distance
  uint32_t bytes;   // bytes of the range
  uint32_t what;    // kMore: another range of the same list follows; kLast: the chunk's last batch;
                    // kStored: no tokens, but bytes of a stored block; kRepeat: all bytes from one distance
};
enum : uint32_t { kMore = 1, kLast = 2, kStored = 4, kRepeat = 8 };

// 256 output bytes: word 32 i + l is the low half of byte 32 i + l's token.
constexpr uint32_t kSteps = 8;
struct ByteBatch {
  uint16_t word[32 * kSteps];
  uint32_t bytes;
  uint32_t near;  // 0: every source lies before the batch; else one more than the bytes before the
                  // first token that starts in the batch; or kStoredBytes, kRepeatedBytes
  uint32_t from;  // kStoredBytes: where they are in the stream; kRepeatedBytes: the distance
  uint32_t last;  // the chunk's last batch; kBadChunk with it if the tokens were not sound
};
constexpr uint32_t kBadChunk = 2, kStoredBytes = 0xffffffffu, kRepeatedBytes = 0xfffffffeu;

using InflateRing = InRing<8>;   // the scan's input
using TokenRing = InRing<2>;     // a token warp's, which lags by up to two stretches
constexpr uint32_t align16(uint32_t v) { return (v + 15u) & ~15u; }
using InflateWin = OutRing<15, 11, true>;  // 32 KiB window, 2 KiB drains by TMA bulk stores
constexpr uint32_t kTeamWarps = 6;

// Shared memory of one team; three teams fit an SM.
struct InflateTeam {
  alignas(128) uint8_t win[InflateWin::kBytes];
  alignas(16) uint8_t ring[align16(InflateRing::kAlloc)];
  alignas(16) uint8_t token_ring[2][align16(TokenRing::kAlloc)];
  InflateTables tab[2];  // the scan warps build the next block's while the token warps read the last's
  ScanBatch batch[2];
  alignas(16) uint32_t tok[2][2][kTokens];  // two lists and two batches per token warp
  TokenBatch out[2][2];
  ByteBatch place[2];
  uint16_t cell_end[2][kPieces];
  uint8_t lens[320];
  uint32_t fill[2][16];
  uint32_t last[kPieces];  // scan warps: where each piece ended, and how
  uint8_t how[kPieces];
  uint32_t redo[2], stop_at[2], sum[2], header_ok;
  int32_t scan_st;
  int32_t status;      // the scan's, with the last token batch
  uint32_t stop;       // set by the place warp: the output is full or a distance is bad
  uint32_t dead;       // a token warp's wait for its input ran out
  uint32_t stopped[2]; // `stop` as the first token warp saw it, one word per batch buffer
  uint64_t bar[8], token_bar[2][2];
};
static_assert(sizeof(InflateTeam) <= 76800, "three teams per SM: 228 KiB / 3 less 1 KiB each");

template <uint32_t ID, uint32_t THREADS>
__device__ __forceinline__ void team_barrier() {
  asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(THREADS) : "memory");
}
template <uint32_t THREADS>
__device__ __forceinline__ void team_wait(uint32_t id) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(THREADS) : "memory");
}
template <uint32_t THREADS>
__device__ __forceinline__ void team_signal(uint32_t id) {  // arrives without waiting
  __threadfence_block();
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(THREADS) : "memory");
}
__device__ __forceinline__ void scan_barrier() { team_barrier<1, 64>(); }                    // the scan warps
__device__ __forceinline__ void batch_barrier() { team_barrier<2, 128>(); }                  // scan -> tokens
// buffer k of a producer and a consumer warp is full (the producer signals) or free (the consumer does);
// batch k of token warp w is 2 w + k
enum : uint32_t { kTokensFull = 4, kTokensFree = 8, kBytesFull = 12, kBytesFree = 14 };

// One symbol, with its distance if it is a length, or two literals.
struct Symbol {
  uint32_t e, d;   // table entries; d is 0 unless e is a length
  uint32_t used;   // bits taken in all
  uint32_t lo, x;  // stream bits of the literal/length and of the distance code
  // end of block, or not a symbol: the table entry's kind has its upper bit set
  __device__ __forceinline__ bool special() const { return ((e | d) & kKindEndBits) != 0; }
  __device__ __forceinline__ bool end() const { return (e & kKindMask) == kKindEndBits; }
  __device__ __forceinline__ bool literal() const { return (e & kKindMask) == kKindLitBits; }
  __device__ __forceinline__ uint32_t count() const { return (e & kPairFlag) ? 2u : 1u; }
  // token of a length and its distance
  __device__ __forceinline__ uint32_t match() const {
    const uint32_t ln = (e >> 5) & 15u, dn = (d >> 5) & 15u;
    return (e & 0xffff0000u) + (bfe32(lo, ln, (e & 31u) - ln) << 16) + (d >> 16) + bfe32(x, dn, (d & 31u) - dn);
  }
};

// Table entries of a symbol with a code longer than its table (or no code: kKindBadBits).
static __device__ __noinline__ uint2 slow_symbol(uint32_t lo, uint32_t hi, InflateTables* tab) {
  uint32_t e = tab->lit_lut[lo & ((1u << kLitLB) - 1u)], d = 0;
  if (e & kSlowFlag) e = slow_entry<kLitLB>(lo, tab->lit(), kAlphaLitLen);
  if ((e & kKindMask) == kKindLenBits) {
    const uint32_t x = __funnelshift_r(lo, hi, e & 31u);
    d = tab->dist_lut[x & ((1u << kDistLB) - 1u)];
    if (d & kSlowFlag) d = slow_entry<kDistLB>(x, tab->dist(), kAlphaDist);
  }
  return make_uint2(e, d);
}

// The symbol whose bits begin `lo`, `hi`.  The distance is looked up whether or not the symbol is a
// length: nearly every time some lane has one, and without a branch several symbols overlap.
__device__ __forceinline__ Symbol symbol(uint32_t lo, uint32_t hi, uint32_t s_lit, uint32_t s_dist, InflateTables& tab) {
  Symbol y;
  y.lo = lo;
  y.e = ld_s32(s_lit + 4u * (lo & ((1u << kLitLB) - 1u)));
  y.x = __funnelshift_r(lo, hi, y.e & 31u);
  const uint32_t d = ld_s32(s_dist + 4u * (y.x & ((1u << kDistLB) - 1u)));
  y.d = (y.e & kKindMask) == kKindLenBits ? d : 0u;
  if ((y.e | y.d) & kSlowFlag) {
    const uint2 z = slow_symbol(lo, hi, &tab);
    y.e = z.x;
    y.d = z.y;
    y.x = __funnelshift_r(lo, hi, y.e & 31u);
  }
  y.used = (y.e & 31u) + (y.d & 31u);
  return y;
}

// inclusive prefix sum over the lanes
__device__ __forceinline__ uint32_t warp_scan_add(uint32_t v, uint32_t lane) {
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t o = __shfl_up_sync(FULL, v, d);
    if (lane >= static_cast<uint32_t>(d)) v += o;
  }
  return v;
}

// ---------------------------------------------------------------------------------------
// scan warps
// ---------------------------------------------------------------------------------------
enum : uint32_t { kRun = 0, kEob = 1, kBad = 2, kFull = 3 };  // how a lane's piece ended

struct InflateScan {
  InflateRing in;  // warp 0 of the two fills it
  InflateTeam& sm;
  uint32_t warp, lane, id;
  uint32_t pos;    // next bit of the stream, in ring coordinates (streams are < 2^28 bytes)
  uint32_t hi8;    // first bit past the stream
  uint32_t span;   // words per piece
  uint32_t k;      // batch buffer
  uint32_t tab, handed;  // tables of this block, and of the batch handed over last
  uint32_t fixed;  // bit t: tab[t] holds the fixed codes

  // 32 stream bits at bit p (they must be resident, or beyond the stream's end)
  __device__ __forceinline__ uint32_t peek(uint32_t p) const {
    const uint32_t a = (p >> 5) << 2;
    return __funnelshift_r(in.rd32(a), in.rd32(a + 4), p & 31u);
  }

  // makes `bits` bits from pos resident (as far as the stream goes); both warps are done reading
  // what lies below pos
  __device__ __forceinline__ int need(uint32_t bits) {
    scan_barrier();
    if (warp == 0) {
      const uint32_t p = pos >> 3, end = ((pos + bits) >> 3) + 8u;
      const int st = in.release(p < in.hi ? p : in.hi) ? in.ensure(end < in.hi ? end : in.hi) : CODAG_ETIMEOUT;
      if (lane == 0) sm.scan_st = st;
    }
    scan_barrier();
    return sm.scan_st;
  }

  // hands batch buffer k to the token warps; false when the place warp wants no more
  __device__ __forceinline__ bool handoff(uint32_t kind, uint32_t base, uint32_t size, int status) {
    if (id == 0) {
      ScanBatch& b = sm.batch[k];
      b.kind = kind;
      b.base = base;
      b.size = size;
      b.table = tab;
      b.status = status;
    }
    batch_barrier();
    const bool go = sm.stopped[k] == 0;
    k ^= 1u;
    handed = tab;
    return go;
  }

  __device__ __forceinline__ Symbol at(uint32_t p, uint32_t s_lit, uint32_t s_dist) const {
    const uint32_t a = in.sbuf + ((p >> 3) & (InflateRing::kMask & ~3u));
    const uint32_t w0 = ld_s32(a), w1 = ld_s32(a + 4), w2 = ld_s32(a + 8), sh = p & 31u;
    return symbol(__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh), s_lit, s_dist, sm.tab[tab]);
  }

  // Where the first symbol that ends at or past `end` ends, decoding from bit p, a guess; what the
  // stream does not allow is stepped over.
  __device__ __forceinline__ uint32_t warm_up(uint32_t p, uint32_t end, bool go, uint32_t s_lit, uint32_t s_dist) {
    while (__any_sync(FULL, go)) {
      if (go) {
        const Symbol y = at(p, s_lit, s_dist);
        p += y.special() ? 1u : y.used;
        go = p < end;
      }
    }
    return p;
  }

  // The symbols of one piece from bit p until one ends at or past `end`, as the serial decoder would
  // read them; every kCell-th start is noted in `row` as an offset from bit `from`.  Every turn brings
  // the lanes back together.
  __device__ __forceinline__ uint32_t piece(uint32_t p, uint32_t end, uint32_t from, bool on, uint16_t* row,
                                            uint32_t s_lit, uint32_t s_dist, uint32_t& cnt, uint32_t& how) {
    uint32_t noted = 0, h = kRun;
    int32_t due = 0;  // symbols before the next start to note
    bool go = on && p < end;
    while (__any_sync(FULL, go)) {
      if (go) {
        const Symbol y = at(p, s_lit, s_dist);
        if (due <= 0) {
          row[noted++] = static_cast<uint16_t>((p - from) | (due < 0 ? 0x8000u : 0u));
          due += kCell;
        }
        p += y.used;
        if (y.special()) {
          h = y.end() ? kEob : kBad;
          go = false;
        } else {
          due -= y.count();
          go = p < end;
          if (go && due <= 0 && noted == kCells) {
            h = kFull;
            go = false;
          }
        }
      }
    }
    cnt = (noted * kCell - due) | (noted << 8);
    if (p > hi8) {  // ran past the end of the stream: no symbol of this piece is taken
      h = kBad;
      cnt = 0;
    }
    how = h;
    return p;
  }

  // The symbols of one block, stretch by stretch, up to and including its end-of-block code.
  __device__ __forceinline__ int symbols() {
    const uint32_t s_lit = smem_u32(sm.tab[tab].lit_lut), s_dist = smem_u32(sm.tab[tab].dist_lut);
    for (;;) {
      // no longer than the rest of the stream needs, so that short streams use all lanes
      const uint32_t rest = (hi8 - pos) / (32u * kPieces), most = rest > kMinSpan ? rest : kMinSpan;
      const uint32_t words = (span < most ? span : most) | 1u;
      const uint32_t bits = words * 32u;
      int st = need(kPieces * bits + 64u);
      if (st) return st;
      // no more symbols than a piece aims at, where they are short
      const uint32_t warm = 32u * span < kWarmBits ? 32u * span : kWarmBits;
      const uint32_t from = pos + id * bits, end = from + bits;
      uint16_t* row = sm.batch[k].row + id * kCells;
      const bool inside = from < hi8;
      uint32_t start = warm_up(id * bits > warm ? from - warm : pos, from, inside && id, s_lit, s_dist);
      if (!inside) start = from;
      bool redo = start < hi8;
      uint32_t last = start, cnt = 0, how = redo ? kRun : kBad;
      uint64_t stop;
      for (;;) {
        uint32_t c, h;
        const uint32_t l = piece(start, end, from, redo, row, s_lit, s_dist, c, h);
        if (redo) {
          last = l;
          cnt = c;
          how = h;
        }
        sm.last[id] = last;
        sm.how[id] = static_cast<uint8_t>(how);
        scan_barrier();
        // lanes whose start is not where the lane below ended; only those below the first lane that
        // ended the stretch matter
        const uint32_t below = id ? sm.last[id - 1] : 0u, bhow = id ? sm.how[id - 1] : static_cast<uint32_t>(kBad);
        redo = bhow == kRun && below != start;
        const uint32_t rm = __ballot_sync(FULL, redo), sp = __ballot_sync(FULL, how != kRun);
        if (lane == 0) {
          sm.redo[warp] = rm;
          sm.stop_at[warp] = sp;
        }
        scan_barrier();
        const uint64_t m = (static_cast<uint64_t>(sm.redo[1]) << 32) | sm.redo[0];
        stop = (static_cast<uint64_t>(sm.stop_at[1]) << 32) | sm.stop_at[0];
        if (!m || (stop && __ffsll(stop) < __ffsll(m))) break;
        if (redo) {
          start = last = below;
          cnt = 0;
          redo = start < hi8;
          how = redo ? kRun : kBad;
        }
      }
      const uint32_t top = stop ? static_cast<uint32_t>(__ffsll(stop)) - 1u : kPieces - 1u;  // last piece that counts
      if (id > top) cnt = 0;
      sm.batch[k].cnt[id] = static_cast<uint16_t>(cnt);
      const uint32_t s = __reduce_add_sync(FULL, cnt & 0xffu);
      if (lane == 0) sm.sum[warp] = s;
      const uint32_t next = sm.last[top], end_how = sm.how[top];
      scan_barrier();
      const uint32_t total = sm.sum[0] + sm.sum[1];
      if (total && !handoff(kBatchTokens, pos, bits, CODAG_OK)) return CODAG_ECORRUPT;
      if (end_how == kBad) return CODAG_ECORRUPT;
      if (total) {
        const uint32_t w = (next - pos) * kPieceTokens / (32u * total);
        span = w < kMaxSpan ? w : kMaxSpan;
      }
      pos = next;
      if (end_how == kEob) return CODAG_OK;
    }
  }

  // Stored block: the copy warp reads its bytes itself, and the ring goes on behind it.
  __device__ __forceinline__ int stored() {
    pos = (pos + 7u) & ~7u;
    int st = need(64);
    if (st) return st;
    const uint32_t v = peek(pos);
    pos += 32;
    const uint32_t len = v & 0xffffu;
    if (len != (~(v >> 16) & 0xffffu)) return CODAG_ECORRUPT;
    if ((pos >> 3) + len > in.hi) return CODAG_ECORRUPT;
    if (len && !handoff(kBatchStored, pos >> 3, len, CODAG_OK)) return CODAG_ECORRUPT;
    pos += len * 8u;
    scan_barrier();
    if (warp == 0 && !in.skip(pos >> 3) && lane == 0) sm.scan_st = CODAG_ETIMEOUT;
    scan_barrier();
    return sm.scan_st;
  }

  // Code lengths and tables of a dynamic block (zlib.h:607-707); both warps read the code lengths,
  // then one builds the literal/length table and the other the distance table.
  __device__ __forceinline__ int dynamic_header() {
    int st = need(2400);  // the largest header: 14 + 19 * 3 + 316 * 7 bits
    if (st) return st;
    const uint32_t v = peek(pos);
    const uint32_t hlit = (v & 31u) + 257u, hdist = ((v >> 5) & 31u) + 1u, hclen = ((v >> 10) & 15u) + 4u;
    pos += 14;
    if (hlit > 286 || hdist > 30) return CODAG_ECORRUPT;
    const HuffTable cl = sm.tab[tab].dist();
    const uint32_t s_cl = smem_u32(sm.tab[tab].dist_lut);
    if (warp == 0) {
      if (lane < 19)  // code length code lengths, 3 bits each in kCodeLenOrder order
        sm.lens[kCodeLenOrder[lane]] = lane < hclen ? static_cast<uint8_t>(peek(pos + 3u * lane) & 7u) : 0;
      __syncwarp();
      const bool ok = order_codes(sm.lens, 19, cl, sm.fill[0], lane);
      __syncwarp();
      if (ok) fill_table<kCodeLenLB, kAlphaCodeLen>(cl, lane, 32);
      __syncwarp();
      for (uint32_t s = lane; s < 80; s += 32) reinterpret_cast<uint32_t*>(sm.lens)[s] = 0;
      if (lane == 0) sm.header_ok = ok;
    }
    pos += 3u * hclen;
    scan_barrier();
    if (!sm.header_ok) return CODAG_ECORRUPT;
    // Literal/length and distance code lengths, run-length coded with symbols 16..18.  Lane l decodes at
    // bit l of a 32-bit stretch; following the lanes' steps from lane 0 by doubling finds the lanes that
    // hold symbols, and a prefix sum of their runs where each run goes.
    uint32_t idx = 0, prev = 0;
    const uint32_t total = hlit + hdist;
    while (idx < total) {
      if (pos > hi8) return CODAG_ECORRUPT;
      const uint32_t bits = peek(pos + lane);
      const uint32_t e = ld_s32(s_cl + 4u * (bits & ((1u << kCodeLenLB) - 1u)));
      const uint32_t n = e & 31u, sym = e >> 16, x = bits >> n;
      const uint32_t rep = sym < 16 ? 1u : sym == 16 ? 3u + (x & 3u) : sym == 17 ? 3u + (x & 7u) : 11u + (x & 127u);
      const uint32_t took = n + (sym < 16 ? 0u : sym == 16 ? 2u : sym == 17 ? 3u : 7u);
      const bool bad = (e & kSlowFlag) != 0;  // code lengths are at most 7 bits
      // lanes reached from lane 0: those of `mask` step to `mask` shifted by their steps, once, twice, four times ...
      uint32_t next = bad ? 63u : lane + took, mask = 1u;
#pragma unroll
      for (int d = 0; d < 5; d++) {
        const uint32_t to = ((mask >> lane) & 1u) && next < 32u ? 1u << next : 0u;
        mask |= __reduce_or_sync(FULL, to);
        const uint32_t further = __shfl_sync(FULL, next, next & 31u);
        next = next < 32u ? further : next;
      }
      const bool here = (mask >> lane) & 1u;
      const uint32_t mine = here && !bad ? rep : 0u, first = idx + warp_scan_add(mine, lane) - mine;
      const bool on = here && first < total;  // symbols past the last length belong to the data
      if (__any_sync(FULL, on && (bad || first + rep > total || (sym == 16 && first == 0)))) return CODAG_ECORRUPT;
      // a repeat takes the value of the last symbol below that is none, else the last stretch's
      const uint32_t own = sym < 16 ? sym : 0u;
      const uint32_t below = __ballot_sync(FULL, here && sym != 16) & lanemask_lt(lane);
      const uint32_t from = __shfl_sync(FULL, own, below ? 31 - __clz(below) : 0);
      const uint32_t val = sym == 16 ? (below ? from : prev) : own;
      if (warp == 0 && on && val)  // a run of more than 6 is zeros
        for (uint32_t t = 0; t < rep; t++) sm.lens[first + t] = static_cast<uint8_t>(val);
      const uint32_t used = __ballot_sync(FULL, on);
      const int last = 31 - __clz(used);
      idx = __shfl_sync(FULL, first + rep, last);
      prev = __shfl_sync(FULL, val, last);
      pos += __shfl_sync(FULL, lane + took, last);
    }
    scan_barrier();
    if (sm.lens[256] == 0) return CODAG_ECORRUPT;
    return build_tables(hlit, sm.lens + hlit, hdist) ? CODAG_OK : CODAG_ECORRUPT;
  }

  // Tables of literal/length codes lens[0..hlit) and distance codes dlens[0..hdist): each warp orders one
  // alphabet, then both fill.
  __device__ __forceinline__ bool build_tables(uint32_t hlit, const uint8_t* dlens, uint32_t hdist) {
    InflateTables& t = sm.tab[tab];
    const bool ok = order_codes(warp ? dlens : sm.lens, warp ? hdist : hlit, warp ? t.dist() : t.lit(), sm.fill[warp], lane);
    if (lane == 0) sm.sum[warp] = ok;
    scan_barrier();
    if (!(sm.sum[0] & sm.sum[1])) return false;
    fill_table<kLitLB, kAlphaLitLen>(t.lit(), id, 64);
    fill_table<kDistLB, kAlphaDist>(t.dist(), id, 64);
    scan_barrier();
    pair_literals<kLitLB>(t.lit_lut, id, 64);
    scan_barrier();
    return true;
  }

  // fixed Huffman codes (RFC 1951 3.2.6)
  __device__ __forceinline__ void fixed_tables() {
    for (uint32_t s = id; s < 320; s += 64) sm.lens[s] = s < 144 ? 8 : s < 256 ? 9 : s < 280 ? 7 : s < 288 ? 8 : 5;
    scan_barrier();
    build_tables(288, sm.lens + 288, 30);
  }

  // The stream bound to `in`, `wrapper` header bytes first.
  __device__ __forceinline__ int run(uint32_t wrapper) {
    if (in.lo + wrapper > in.hi) return CODAG_ECORRUPT;
    pos = (in.lo + wrapper) * 8u;
    hi8 = in.hi * 8u;
    span = kMaxSpan;
    bool last = false;
    while (!last) {
      if (pos >= hi8) return CODAG_ECORRUPT;
      int st = need(64);
      if (st) return st;
      const uint32_t h = peek(pos);
      last = h & 1u;
      const uint32_t btype = (h >> 1) & 3u;
      pos += 3;
      tab = handed ^ 1u;  // the token warps may still read the tables of the last batch
      if (btype == 0) {
        st = stored();
      } else if (btype == 1) {
        if (!((fixed >> tab) & 1u)) fixed_tables();
        fixed |= 1u << tab;
      } else if (btype == 2) {
        fixed &= ~(1u << tab);
        st = dynamic_header();
      } else {
        st = CODAG_ECORRUPT;
      }
      if (!st && btype) st = symbols();
      if (st) return st;
    }
    return pos > hi8 ? CODAG_ECORRUPT : CODAG_OK;
  }
};

// Binds a warp's input ring (it initialises the barriers) and the window of a team.
template <int NSLOT>
__device__ __forceinline__ void bind_ring(InRing<NSLOT>& in, uint8_t* buf, uint64_t* bar, uint64_t wait_cycles,
                                          uint32_t lane, bool init) {
  in.buf = buf;
  in.sbuf = smem_u32(buf);
  in.bar = bar;
  in.phase = 0;
  in.wait_cycles = wait_cycles;
  in.lane = lane;
  if (init) init_ring_barriers<NSLOT>(bar, lane);
}
__device__ __forceinline__ void inflate_rings(InflateRing& in, TokenRing& tin, InflateTeam& sm, uint64_t wait_cycles,
                                              uint32_t warp, uint32_t lane) {
  bind_ring(in, sm.ring, sm.bar, wait_cycles, lane, warp == 0);
  const uint32_t w = warp & 1u;
  bind_ring(tin, sm.token_ring[w], sm.token_bar[w], wait_cycles, lane, (warp >> 1) == 1);
}
__device__ __forceinline__ void inflate_window(InflateWin& o, InflateTeam& sm, uint32_t lane) {
  o.buf = sm.win;
  o.sbuf = smem_u32(sm.win);
  o.lane = lane;
}

// Scan warps (0 and 1 of the team): the stream bound to `in`.
__device__ __forceinline__ void inflate_scan(InflateRing& in, InflateTeam& sm, uint32_t wrapper, uint32_t warp,
                                             uint32_t lane) {
  InflateScan d{in, sm, warp, lane, warp * 32u + lane, 0, 0, 0, 0, 0, 1, 0};
  int st = d.run(wrapper);
  if (warp == 0) {
    if (!d.in.drain()) st = CODAG_ETIMEOUT;
    in.phase = d.in.phase;  // the next stream through this ring goes on from here
  }
  d.handoff(kBatchDone, 0, 0, st);
}

// ---------------------------------------------------------------------------------------
// token warps
// ---------------------------------------------------------------------------------------
// Token warps (2 and 3 of the team: `me` 0 and 1), taking turns at 32 cells or a stored block; `in`
// is bound to the stream.  Every turn ends in a batch, an empty one when no more are wanted, so the
// place warp knows whose turn it is.
__device__ __forceinline__ void inflate_tokens(TokenRing& in, InflateTeam& sm, uint32_t me, uint32_t lane) {
  uint32_t kb = 0, turn = 0, list = 0, k = 0, used = 0;
  const auto reuse = [&]() {  // waits until the place warp is done with the batch before last, and its list
    if (used >= 2u) team_wait<64>(kTokensFree + 2u * me + k);
    used++;
  };
  const auto handoff = [&](uint32_t before, uint32_t bytes, uint32_t what) {
    if (lane == 0) {
      TokenBatch& o = sm.out[me][k];
      o.list = list;
      o.before = before;
      o.bytes = bytes;
      o.what = what;
    }
    __syncwarp();
    team_signal<64>(kTokensFull + 2u * me + k);
    k ^= 1u;
    if (!(what & kMore)) list ^= 1u;
  };
  // the place warp's word, the same for every lane
  const auto stopped = [&]() {
    const uint32_t v = *static_cast<volatile uint32_t*>(&sm.stop) | *static_cast<volatile uint32_t*>(&sm.dead);
    return __shfl_sync(FULL, v, 0) != 0;
  };
  // bytes [at, end) resident
  const auto need = [&](uint32_t at, uint32_t end) {
    const bool ok = in.release(at) && in.ensure(end < in.hi ? end : in.hi) == CODAG_OK;
    if (!ok && lane == 0) sm.dead = 1;
    return ok;
  };
  for (;;) {
    if (me == 0) {
      const bool drop = stopped();
      if (lane == 0) sm.stopped[kb] = drop;  // both scan warps read the word of their batch's buffer
    }
    batch_barrier();
    ScanBatch& b = sm.batch[kb];
    kb ^= 1u;
    const uint32_t kind = b.kind;
    if (kind == kBatchDone) {
      const bool drained = in.drain();
      if (!drained && lane == 0) sm.dead = 1;
      if ((turn & 1u) == me) {
        if (lane == 0) sm.status = b.status;
        reuse();
        handoff(0, 0, kLast);
      }
      if (used >= 2u) team_wait<64>(kTokensFree + 2u * me + k);
      if (used) team_wait<64>(kTokensFree + 2u * me + (k ^ 1u));
      return;
    }
    if (kind == kBatchStored) {
      if ((turn++ & 1u) == me) {
        reuse();
        const bool drop = stopped();
        handoff(b.base, drop ? 0u : b.size, drop ? 0u : static_cast<uint32_t>(kStored));
      }
      if (!in.skip(b.base + b.size) && lane == 0) sm.dead = 1;
      continue;
    }
    // cells of the pieces, as running totals
    uint16_t* cell_end = sm.cell_end[me];
    const uint32_t e0 = warp_scan_add(b.cnt[lane] >> 8, lane);
    const uint32_t e1 = warp_scan_add(b.cnt[32 + lane] >> 8, lane) + __shfl_sync(FULL, e0, 31);
    const uint32_t cells = __shfl_sync(FULL, e1, 31);
    cell_end[lane] = static_cast<uint16_t>(e0);
    cell_end[32 + lane] = static_cast<uint16_t>(e1);
    __syncwarp();
    InflateTables& tab = sm.tab[b.table];
    const uint32_t s_lit = smem_u32(tab.lit_lut), s_dist = smem_u32(tab.dist_lut);
    const uint32_t base = b.base, bits = b.size;
    for (uint32_t c = 0; c < cells; c += 32, turn++) {
      if ((turn & 1u) != me) continue;
      const uint32_t count = cells - c < 32u ? cells - c : 32u;
      const uint32_t x = c + (lane < count ? lane : count - 1u);  // lanes past the end repeat the last cell
      uint32_t q = 0;  // its piece: as many as end at or before it
#pragma unroll
      for (uint32_t step = kPieces / 2; step; step >>= 1)
        if (cell_end[q + step - 1u] <= x) q += step;
      const uint32_t first = q ? cell_end[q - 1u] : 0u, j = x - first;
      const uint16_t* row = b.row + q * kCells + j;
      uint32_t p = base + q * bits + (row[0] & 0x7fffu);
      const uint32_t next = j + 1u < b.cnt[q] >> 8 ? kCell * (j + 1u) + (row[1] >> 15) : b.cnt[q] & 0xffu;
      const uint32_t n = lane < count ? next - (kCell * j + (row[0] >> 15)) : 0u;
      uint32_t* dst = sm.tok[me][list] + (warp_scan_add(n, lane) - n);
      uint32_t len = 0;  // bytes of this lane's tokens
      reuse();
      bool ok = !stopped();
      // as many of the cells, which follow one another, at a time as the ring holds for certain:
      // mostly all
      for (uint32_t l0 = 0; ok && l0 < count;) {
        constexpr uint32_t kCellBits = 48u * kCellMax + 96u;
        const uint32_t p0 = __shfl_sync(FULL, p, static_cast<int>(l0));
        const uint32_t fit = __ballot_sync(FULL, lane >= l0 && p - p0 + kCellBits <= 8u * kSlotBytes);
        const uint32_t l1 = fit ? 32u - __clz(fit) : l0;  // [l0, l1): the cells that fit
        const uint32_t last = __shfl_sync(FULL, p, static_cast<int>(l1) - 1);
        ok = l1 > l0 && need(p0 >> 3, (last + kCellBits) >> 3);
        if (!ok) break;
        const bool mine = lane >= l0 && lane < l1;
        for (uint32_t i = 0; __any_sync(FULL, mine && i < n);) {
          if (mine && i < n) {
            const uint32_t a = in.sbuf + ((p >> 3) & (TokenRing::kMask & ~3u));
            const uint32_t w0 = ld_s32(a), w1 = ld_s32(a + 4), w2 = ld_s32(a + 8), sh = p & 31u;
            const Symbol y = symbol(__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh), s_lit, s_dist, tab);
            const uint32_t tok = y.literal() ? kLiteralToken | ((y.e >> 16) & 0xffu) : y.match();
            dst[i] = tok;
            if (y.e & kPairFlag) dst[i + 1u] = kLiteralToken | (y.e >> 24);
            len += (tok >> 16) + y.count() - 1u;
            i += y.count();
            p += y.used;
          }
        }
        l0 = l1;
      }
      if (!ok) {
        handoff(0, 0, 0);
        continue;
      }
      uint32_t s0 = warp_scan_add(len, lane);
      const uint32_t total = __shfl_sync(FULL, s0, 31);
      s0 -= len;
      if (total == 0) {  // a single cell noted just before the end of its block
        handoff(0, 0, 0);
        continue;
      }
      // bytes [r, r + bytes) of the list: a mark where each token starts
      const auto mark = [&](uint32_t r, uint32_t bytes) {
        uint32_t* starts = sm.out[me][k].starts;
        for (uint32_t i = lane; i < kRange / 32u; i += 32) starts[i] = 0;
        __syncwarp();
        uint32_t s = s0, before = 0;
        if (total <= kRange) {
#pragma unroll 4
          for (uint32_t i = 0; i < n; i++) {
            const uint32_t tok = dst[i];
            atomicOr(&starts[s >> 5], 1u << (s & 31u));
            s += tok >> 16;
          }
        } else {
          for (uint32_t i = 0; i < n; i++) {
            const uint32_t tok = dst[i];
            if (s < r) before++;
            else if (s - r < bytes) atomicOr(&starts[(s - r) >> 5], 1u << ((s - r) & 31u));
            s += tok >> 16;
          }
          before = __reduce_add_sync(FULL, before);
        }
        handoff(before, bytes, r + bytes < total ? kMore : 0u);
      };
      if (total <= kRange) {
        mark(0, total);
        continue;
      }
      // Long matches: lanes whose tokens all have one distance, and neighbours at the same, go as one batch; the
      // bytes of the others in ranges the bit map covers.
      constexpr uint32_t kRepeatMin = 512;  // bytes of a lane's tokens
      uint32_t dist = n && len >= kRepeatMin ? dst[0] & 0xffffu : kLiteral;
      if (!(dist >> 15))
        for (uint32_t i = 1; i < n; i++)
          if ((dst[i] & 0xffffu) != dist) dist = kLiteral;
      if (dist >> 15) dist = kLiteral;
      const uint32_t below = __shfl_up_sync(FULL, dist, 1);
      uint32_t cuts = __ballot_sync(FULL, lane == 0 || dist != below);
      bool again = false;
      while (cuts) {
        const uint32_t a = __ffs(cuts) - 1u;
        cuts &= cuts - 1u;
        const uint32_t x = __shfl_sync(FULL, s0, a), d = __shfl_sync(FULL, dist, a);
        const uint32_t next = __shfl_sync(FULL, s0, cuts ? __ffs(cuts) - 1 : 0), y = cuts ? next : total;
        if (d == kLiteral) {
          for (uint32_t r = x; r < y; r += kRange) {
            if (again) reuse();
            again = true;
            mark(r, y - r < kRange ? y - r : kRange);
          }
        } else {
          if (again) reuse();
          again = true;
          handoff(d + 1u, y - x, kRepeat | (y < total ? kMore : 0u));
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------------------
// place warp
// ---------------------------------------------------------------------------------------
// Warp 4 of the team: the token word of every output byte.  Stops the chunk when its output would pass
// `cap` or a distance reaches before its first byte.
__device__ __forceinline__ void inflate_place(InflateTeam& sm, uint64_t chunk_bytes, uint32_t lane) {
  const uint32_t cap = static_cast<uint32_t>(chunk_bytes);
  const uint32_t le = 0xffffffffu >> (31u - lane);
  uint32_t op = 0, me = 0, from = 0, k = 0, handed = 0;  // from: bit w, the batch token warp w fills next
  bool ok = true;
  const auto handoff = [&](uint32_t bytes, uint32_t near, uint32_t last) {
    if (lane == 0) {
      sm.place[k].bytes = bytes;
      sm.place[k].near = near;
      sm.place[k].last = last;
    }
    __syncwarp();
    team_signal<64>(kBytesFull + k);
    k ^= 1u;
    handed++;
  };
  for (;;) {
    const uint32_t buf = (from >> me) & 1u;
    team_wait<64>(kTokensFull + 2u * me + buf);
    const TokenBatch& b = sm.out[me][buf];
    const uint32_t bytes = b.bytes, what = b.what, s_tok = smem_u32(sm.tok[me][b.list]);
    if (bytes > cap - op) ok = false;
    constexpr uint32_t kWhole = kStored | kRepeat;
    if ((what & kRepeat) && b.before > op) ok = false;
    if (ok && (what & kWhole)) {
      if (handed >= 2u) team_wait<64>(kBytesFree + k);
      if (lane == 0) sm.place[k].from = b.before;
      handoff(bytes, what & kStored ? kStoredBytes : kRepeatedBytes, 0);
    }
    uint32_t count = b.before;  // tokens that start before the 1 KiB at c
    for (uint32_t c = what & kWhole ? bytes : 0u; ok && c < bytes; c += 1024) {
      // lane l: the starts in the 32 bytes at c + 32 l, and how many tokens start before them
      const uint32_t word = c + 32u * lane < bytes ? b.starts[c / 32u + lane] : 0u;
      const uint32_t upto = warp_scan_add(__popc(word), lane) + count, pre = upto - __popc(word);
      count = __shfl_sync(FULL, upto, 31);
      const uint32_t end = bytes - c < 1024u ? bytes - c : 1024u;
      for (uint32_t q = 0; q < end; q += 32 * kSteps) {
        const uint32_t b0 = op + c + q, n = end - q;
        uint32_t w[kSteps], t[kSteps];
        bool near = false;
#pragma unroll
        for (uint32_t i = 0; i < kSteps; i++) {
          const uint32_t starts = __shfl_sync(FULL, word, q / 32u + i);
          t[i] = __shfl_sync(FULL, pre, q / 32u + i) + __popc(starts & le) - 1u;
          // bytes past the end are taken for literals
          w[i] = 32u * i + lane < n ? ld_s16(s_tok + 4u * t[i]) : kLiteral;
          near |= w[i] < 32u * i + lane;
        }
        if (b0 < 32768u) {
          bool bad = false;
#pragma unroll
          for (uint32_t i = 0; i < kSteps; i++) bad |= !(w[i] >> 15) && w[i] >= b0 + 32u * i + lane;
          if (__any_sync(FULL, bad)) {
            ok = false;
            break;
          }
        }
        uint32_t lead = 0;
        if (__any_sync(FULL, near)) {
          const uint32_t some = __ballot_sync(FULL, word != 0) & (FULL << (q / 32u));
          const uint32_t f = some ? __ffs(some) - 1u : 32u;  // the first 32 bytes with a start
          lead = f - q / 32u < kSteps ? 32u * (f - q / 32u) + __ffs(__shfl_sync(FULL, word, f & 31u)) - 1u : 32u * kSteps;
          lead++;
          bool inside = false;
#pragma unroll
          for (uint32_t i = 0; i < kSteps; i++) inside |= w[i] < lane;
          if (lead <= n && __any_sync(FULL, inside)) {
            // Sources among a step's own 32 bytes are followed to a lane that starts outside or is a literal,
            // chains of up to 31 links halved five times, and its word taken over; all steps side by side.
            uint32_t root[kSteps];
#pragma unroll
            for (uint32_t i = 0; i < kSteps; i++) root[i] = w[i] < lane ? lane - 1u - w[i] : lane;
#pragma unroll
            for (int d = 0; d < 5; d++) {
#pragma unroll
              for (uint32_t i = 0; i < kSteps; i++) root[i] = __shfl_sync(FULL, root[i], root[i]);
            }
#pragma unroll
            for (uint32_t i = 0; i < kSteps; i++) {
              const uint32_t v = __shfl_sync(FULL, w[i], root[i]);
              const uint32_t to = v >> 15 ? v : v + (lane - root[i]);
              // a distance past 32768 has no word: the copy warp follows that step's chains itself
              if (!__any_sync(FULL, !(v >> 15) && to >= kLiteral)) w[i] = to;
            }
          }
        }
        if (handed >= 2u) team_wait<64>(kBytesFree + k);
#pragma unroll
        for (uint32_t i = 0; i < kSteps; i++) sm.place[k].word[32u * i + lane] = static_cast<uint16_t>(w[i]);
        handoff(n < 32u * kSteps ? n : 32u * kSteps, lead, 0);
      }
    }
    team_signal<64>(kTokensFree + 2u * me + buf);
    from ^= 1u << me;
    if (ok) op += bytes;
    else if (lane == 0) sm.stop = 1;
    __syncwarp();
    if (what & kLast) break;
    if (!(what & kMore)) me ^= 1u;
  }
  if (handed >= 2u) team_wait<64>(kBytesFree + k);
  handoff(0, 0, ok ? 1u : 1u | kBadChunk);
  // the copy warp's last two signals
  if (handed >= 2u) team_wait<64>(kBytesFree + k);
  team_wait<64>(kBytesFree + (k ^ 1u));
}

// ---------------------------------------------------------------------------------------
// copy warp
// ---------------------------------------------------------------------------------------
// n bytes of the stream (`g`, which ends at `hi`) from `from` on to output position op, 2 KiB at a time: words that lie
// whole in the stream, put together to words of the window, and single bytes around them.  The result: out.flushed.
template <class OUT>
__device__ __noinline__ uint32_t copy_stored(OUT out, uint32_t op, uint32_t n, const uint8_t* __restrict__ g, uint32_t from,
                                         uint32_t hi, uint32_t lane) {
  while (n) {
    const uint32_t room = OUT::kFlush - (op & (OUT::kFlush - 1u)), m = n < room ? n : room;
    const uint32_t ahead = from + 4u * OUT::kFlush + 64u * lane;
    if (ahead < hi) asm volatile("prefetch.global.L2 [%0];" ::"l"(g + ahead));
    const uint32_t head = (0u - op) & 3u, h = head < m ? head : m;
    const uint32_t a0 = (from + h) & ~3u, sh = 8u * ((from + h) & 3u);
    const uint32_t in_stream = a0 + 8u <= hi ? (hi - 8u - a0) / 4u + 1u : 0u;
    const uint32_t words = (m - h) / 4u < in_stream ? (m - h) / 4u : in_stream;
    constexpr uint32_t kEach = 8;
#pragma unroll 1
    for (uint32_t w0 = 0; w0 < words; w0 += 32u * kEach) {
      uint32_t x[kEach], y[kEach];
#pragma unroll
      for (uint32_t i = 0; i < kEach; i++) {
        const uint32_t w = w0 + 32u * i + lane;
        const uint32_t* p = reinterpret_cast<const uint32_t*>(g + a0) + (w < words ? w : words - 1u);
        x[i] = __ldg(p);
        y[i] = __ldg(p + 1);
      }
#pragma unroll
      for (uint32_t i = 0; i < kEach; i++) {
        const uint32_t w = w0 + 32u * i + lane;
        if (w < words) st_s32(out.sbuf + ((op + h + 4u * w) & OUT::kMask), __funnelshift_r(x[i], y[i], sh));
      }
    }
    if (lane < h) out.put8(op + lane, __ldg(g + from + lane));
    for (uint32_t b = h + 4u * words + lane; b < m; b += 32) out.put8(op + b, __ldg(g + from + b));
    __syncwarp();
    op += m;
    from += m;
    n -= m;
    out.flush_to(op);
  }
  return out.flushed;
}

// n bytes at distance d from output position op on, 2 KiB at a time: single bytes from the d before them, and 16 at
// once from a multiple of d and of 16 further back as soon as the repetition reaches that far (zeros: 128 KiB a
// byte a lane 105 us, 16 bytes a lane 20).
template <class OUT>
__device__ __noinline__ uint32_t copy_repeated(OUT out, uint32_t op, uint32_t n, uint32_t d, uint32_t lane) {
  const uint32_t step = 32u % d, far = 16u * d * ((512u + 16u * d - 1u) / (16u * d));
  const auto bytes = [&](uint32_t count) {  // from op on
    uint32_t r = lane % d;
    for (uint32_t at = lane; at - lane < count; at += 128) {
      uint32_t v[4];
#pragma unroll
      for (uint32_t i = 0; i < 4; i++) {
        v[i] = out.get8(op - d + r);
        r += step;
        if (r >= d) r -= d;
      }
      __syncwarp();  // a far source's place is that of a byte written here
#pragma unroll
      for (uint32_t i = 0; i < 4; i++)
        if (at + 32u * i < count) out.put8(op + at + 32u * i, v[i]);
      __syncwarp();
    }
    op += count;
    n -= count;
  };
  const uint32_t start = op - d;  // the repetition goes back to here
  while (n) {
    const uint32_t room = OUT::kFlush - (op & (OUT::kFlush - 1u)), m = n < room ? n : room;
    const uint32_t head = (0u - op) & 15u, body = m > head ? (m - head) & ~15u : 0u;
    if (body && far <= OUT::kBytes / 2 && op + head - start >= far) {
      if (head) bytes(head);
      for (uint32_t w = 16u * lane; w - 16u * lane < body; w += 512) {  // far is at least 512: sources lie before the step
        if (w < body) st_s128(out.sbuf + ((op + w) & OUT::kMask), ld_s128(out.sbuf + ((op + w - far) & OUT::kMask)));
        __syncwarp();
      }
      op += body;
      n -= body;
      if (m - head - body) bytes(m - head - body);
    } else {
      bytes(m);
    }
    out.flush_to(op);
  }
  return out.flushed;
}

// Warp 5 of the team: writes the bytes through `out` and returns the chunk's status.  `src`: the stream.
template <class OUT>
__device__ __forceinline__ int inflate_copy(InflateTeam& sm, OUT& out, const uint8_t* src, uint32_t len, uint32_t lane) {
  const uint32_t lo = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(src) & 15u);  // as in the rings
  uint32_t op = 0, k = 0, last;
  do {
    team_wait<64>(kBytesFull + k);
    const ByteBatch& b = sm.place[k];
    const uint32_t n = b.bytes, near = b.near;
    last = b.last;
    if (!near) {  // every source lies before the batch: all bytes at once
      uint32_t v[kSteps];
#pragma unroll
      for (uint32_t i = 0; i < kSteps; i++) v[i] = b.word[32u * i + lane];
#pragma unroll
      for (uint32_t i = 0; i < kSteps; i++)
        if (!(v[i] >> 15) && 32u * i < n) v[i] = out.get8(op + 32u * i + lane - 1u - v[i]);
      __syncwarp();  // from distance 32513 on a source's place in the window is that of a later byte of the batch
#pragma unroll
      for (uint32_t i = 0; i < kSteps; i++)
        if (32u * i + lane < n) out.put8(op + 32u * i + lane, v[i]);
      __syncwarp();
    } else if (near > n) {
      if (near == kStoredBytes) {
        out.flushed = copy_stored(out, op, n, src - lo, b.from, lo + len, lane);
      } else if (near == kRepeatedBytes) {
        out.flushed = copy_repeated(out, op, n, b.from, lane);
      } else {  // one match, repeating itself
        const uint32_t d = b.word[0] + 1u, step = 32u % d;
        uint32_t r = lane % d;
#pragma unroll 4
        for (uint32_t at = lane; at - lane < n; at += 32) {
          const uint32_t v = out.get8(op - d + r);
          if (at < n) out.put8(op + at, v);
          r += step;
          if (r >= d) r -= d;
        }
        __syncwarp();
      }
    } else {
#pragma unroll 1
      for (uint32_t h = 0; h < n; h += 128) {
        uint32_t v[4];
        bool inside = false;
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) {
          v[i] = b.word[h + 32u * i + lane];
          inside |= v[i] < 32u * i + lane;
        }
        if (!__any_sync(FULL, inside)) {  // every source lies before these 128 bytes
#pragma unroll
          for (uint32_t i = 0; i < 4; i++)
            if (!(v[i] >> 15) && h + 32u * i < n) v[i] = out.get8(op + h + 32u * i + lane - 1u - v[i]);
          __syncwarp();
#pragma unroll
          for (uint32_t i = 0; i < 4; i++)
            if (h + 32u * i + lane < n) out.put8(op + h + 32u * i + lane, v[i]);
          __syncwarp();
          continue;
        }
#pragma unroll 1
        for (uint32_t i = h; i < n && i < h + 128u; i += 32) {
          const uint32_t w = b.word[i + lane];
          uint32_t x = w;
          if (w >= lane && !(w >> 15)) x = out.get8(op + i + lane - 1u - w);
          if (__any_sync(FULL, w < lane)) {
            // follow sources among the 32 to a lane that starts outside or is a literal: chains of up
            // to 31 links, halved five times
            uint32_t root = w < lane ? lane - 1u - w : lane;
#pragma unroll
            for (int j = 0; j < 5; j++) root = __shfl_sync(FULL, root, root);
            x = __shfl_sync(FULL, x, root);
          }
          __syncwarp();
          if (i + lane < n) out.put8(op + i + lane, x);
          __syncwarp();
        }
      }
    }
    team_signal<64>(kBytesFree + k);
    k ^= 1u;
    op += n;
    out.flush_to(op);
  } while (!last);
  out.finish(op);
  if (sm.dead) return CODAG_ETIMEOUT;
  const int st = sm.status;
  if (st != CODAG_OK) return st;
  return !(last & kBadChunk) && op >= out.store ? CODAG_OK : CODAG_ECORRUPT;
}

}  // namespace codag_dev
