// Batched persistent decompression (include/codag.h, codag_batch_*): one launch over many
// independent streams of uneven size and mixed codec.
#include <algorithm>
#include <cstdint>
#include <mutex>
#include <new>
#include <utility>
#include <vector>

#include "capi_common.cuh"
#include "decode_deflate_warp.cuh"
#include "decode_rle_team.cuh"

using namespace codag_dev;
using namespace codag_capi;

namespace {

constexpr uint32_t kWarps = kTeamWarps;  // warps per CTA (eight, for RLE files, cost Deflate 7% in registers)
using RleRing = InRing<4>;
using BatchV2 = TeamV2<3>;
struct OneWarp {  // a stream on one warp
  alignas(128) uint8_t ring[align_up(RleRing::kAlloc, 128)];
  alignas(16) uint8_t win[InflateWarpWin::kBytes];  // Deflate
  InflateWarp tables;
};
struct BatchShared {
  union {
    InflateTeam inflate;
    TeamV1 v1;
    BatchV2 v2;
    OneWarp one[kWarps];
  };
  TeamBars tb;
  uint64_t bar[kWarps][4];  // of the warps' own rings
  uint32_t job;
  uint32_t ahead;  // the next entry for a team, as far as the threads have looked
  int32_t st;
};
static_assert(sizeof(TeamV1) <= offsetof(InflateTeam, bar) && sizeof(BatchV2) <= offsetof(InflateTeam, bar) &&
                  kWarps * sizeof(OneWarp) <= offsetof(InflateTeam, bar),
              "the Deflate team's barriers keep their place");
static_assert(sizeof(BatchShared) <= 76800, "three CTAs per SM");

struct BatchArgs {
  const codag_chunk_desc* descs;
  const uint32_t* order;
  const uint8_t* comp;
  uint64_t comp_bytes;
  uint8_t* out;
  uint64_t out_bytes;
  int32_t* status;
};

__device__ __forceinline__ bool job_in_bounds(const BatchArgs& a, const codag_chunk_desc& d) {
  return d.out_off <= a.out_bytes && d.out_len <= a.out_bytes - d.out_off &&
         stream_in_bounds(d.comp_off, d.comp_len, a.comp_bytes);
}

// A Deflate stream on one warp
__device__ __noinline__ int inflate_job(const uint8_t* src, uint32_t len, uint8_t* dst, uint32_t out_len, uint32_t wrapper,
                                        RleRing& ring, OneWarp& sh, uint32_t lane) {
  RleRing in = ring;
  in.begin(src, len);
  InflateWarpWin o;
  o.buf = sh.win;
  o.sbuf = smem_u32(sh.win);
  o.lane = lane;
  o.begin(dst, out_len);
  const int st = inflate_warp(in, o, sh.tables, out_len, wrapper, lane);
  ring = in;
  return st;
}

// A stream on one warp.  RLE values go straight to global memory: element by element when the
// output is element aligned, byte by byte otherwise.
__device__ __forceinline__ int warp_job(const BatchArgs& a, const codag_chunk_desc& d, RleRing& in, OneWarp& sh, uint32_t lane) {
  if (!job_in_bounds(a, d)) return CODAG_ECORRUPT;
  if (d.codec == CODAG_CODEC_DEFLATE)
    return inflate_job(a.comp + d.comp_off, d.comp_len, a.out + d.out_off, d.out_len, d.wrapper_bytes, in, sh, lane);
  if (d.codec != CODAG_CODEC_RLEV1 && d.codec != CODAG_CODEC_RLEV2) return CODAG_EINVAL;
  in.begin(a.comp + d.comp_off, d.comp_len);
  const uint32_t e = d.elem_bytes;
  if (valid_elem_dev(e) && (reinterpret_cast<uintptr_t>(a.out + d.out_off) % e) == 0 && d.out_len % e == 0) {
    DirectOut od;
    od.lane = lane;
    od.begin(a.out + d.out_off, d.out_len);
    return decode_rle_any(d.codec, in, od, d.out_len, static_cast<int>(e));
  }
  ByteOut ob;
  ob.lane = lane;
  ob.begin(a.out + d.out_off, d.out_len);
  return decode_rle_any(d.codec, in, ob, d.out_len, static_cast<int>(e));
}

__device__ __forceinline__ void rle_ring(RleRing& in, OneWarp& sh, uint64_t* bar, uint64_t wait_cycles, uint32_t lane) {
  in.buf = sh.ring;
  in.sbuf = smem_u32(in.buf);
  in.bar = bar;
  in.phase = 0;
  in.wait_cycles = wait_cycles;
  in.lane = lane;
  init_ring_barriers<4>(in.bar, lane);
}

// An RLE stream on the whole CTA
template <int CODEC, int E, class Team>
__device__ __noinline__ uint32_t rle_team_job(Team& sm, TeamBars& tb, const uint8_t* src, uint32_t len, uint8_t* dst,
                                              uint32_t out_len, uint64_t wait_cycles) {
  return rle_team<CODEC, E, kWarps>(sm, tb, src, len, dst, out_len, out_len / E, wait_cycles);
}
template <int CODEC, class Team>
__device__ __forceinline__ uint32_t rle_team_any(Team& sm, TeamBars& tb, const BatchArgs& a, const codag_chunk_desc& d,
                                                 uint64_t wait_cycles) {
  const uint8_t* src = a.comp + d.comp_off;
  uint8_t* dst = a.out + d.out_off;
  switch (d.elem_bytes) {
    case 8: return rle_team_job<CODEC, 8>(sm, tb, src, d.comp_len, dst, d.out_len, wait_cycles);
    case 4: return rle_team_job<CODEC, 4>(sm, tb, src, d.comp_len, dst, d.out_len, wait_cycles);
    case 2: return rle_team_job<CODEC, 2>(sm, tb, src, d.comp_len, dst, d.out_len, wait_cycles);
    default: return rle_team_job<CODEC, 1>(sm, tb, src, d.comp_len, dst, d.out_len, wait_cycles);
  }
}
__device__ __forceinline__ bool rle_team_takes(const BatchArgs& a, const codag_chunk_desc& d) {
  const uint32_t e = d.elem_bytes;
  return job_in_bounds(a, d) && (d.codec == CODAG_CODEC_RLEV1 || d.codec == CODAG_CODEC_RLEV2) && valid_elem_dev(e) &&
         (reinterpret_cast<uintptr_t>(a.out + d.out_off) % e) == 0 && d.out_len % e == 0 &&
         (d.comp_len | d.out_len) < 0x80000000u;
}

// RLE files below this size, and RLE v2 files of it, are taken by a warp each (3000 RLE v1 files of 32 KiB without a
// plan: 179 us by warps | 143).  So are longer RLE v2 files where there are more of them
// than CTAs are resident (as in codag_decompress_rlev2; 2048 of 128 KiB: 257 us | 581 by CTAs), but for the
// longest: those above the smallest power of two that no more than the resident CTAs exceed, so that a few
// long files among many are not left to single warps (450 of 40 KB and one of 8 MiB: 7.1 ms by warps | 5.3).
constexpr uint32_t kWarpBytes = 32768;
constexpr uint32_t kShifts = 18;  // file sizes are below kWarpBytes << 17
__host__ __device__ __forceinline__ uint32_t shifts_below(uint32_t out_len) {  // how many j have out_len > kWarpBytes << j
  uint32_t j = 0;
  while (out_len > static_cast<uint64_t>(kWarpBytes) << j) j++;
  return j;
}
// long_v2[j]: RLE v2 files for teams with shifts_below of j; the result: those with more than it gives get a CTA
__host__ __device__ __forceinline__ uint32_t v2_shift(const uint32_t* long_v2, uint64_t resident) {
  uint64_t longer = 0;
  uint32_t s = kShifts - 1;
  while (s > 0 && (longer += long_v2[s]) <= resident) s--;
  return s;
}
__host__ __device__ __forceinline__ bool rle_team_pays(const codag_chunk_desc& d, uint32_t shift) {
  if (d.out_len < kWarpBytes || d.comp_len <= kTeamMinBytes) return false;  // (3000 of 40 KB in 120 bytes each: 112 us | 97)
  if (d.codec == CODAG_CODEC_RLEV1) return true;
  // mostly DIRECT groups, if it is that long: see rlev2_alone
  const bool direct = d.comp_len > (2u + d.elem_bytes / 4u) * static_cast<uint64_t>(d.out_len / d.elem_bytes);
  return shifts_below(d.out_len) > shift && !direct;
}

// Deflate files that warps (18 a SM) get through faster than teams (three a SM).  Teams take them all the same where
// these are done before the longest of them is on a warp.
struct InflateJob {
  InflateCost c;
  __host__ __device__ __forceinline__ explicit InflateJob(const codag_chunk_desc& d) : c(inflate_cost(d.out_len, d.comp_len)) {}
  __host__ __device__ __forceinline__ bool small() const { return 15.f * c.team > 4.f * c.warp; }
};
struct SmallInflates {
  float team = 0, longest = 0;
  __host__ __device__ __forceinline__ void add(const InflateJob& j) {
    if (!j.small()) return;
    team += j.c.team;
    longest = longest > j.c.warp ? longest : j.c.warp;
  }
  __host__ __device__ __forceinline__ bool by_warps(uint64_t resident) const { return team > longest * static_cast<float>(resident); }
};

// Without a plan the host does not know the files.  k_classify writes to *queue what k_batch has to know of
// them; k_batch counts its entries in the low bits.  It goes over the list twice: CTAs take the files for
// teams, then single warps the others, which is how a plan sorts them.
constexpr uint32_t kCountBits = 25, kAnyTeam = 1u << 31, kInflateWarps = 1u << kCountBits, kShiftAt = kCountBits + 1;
constexpr uint64_t kMaxMixed = (1u << (kCountBits - 1)) - 65536u;  // counts to twice that, and once more per warp
__device__ __forceinline__ bool wants_team(const BatchArgs& a, const codag_chunk_desc& d, uint32_t flags) {
  if (d.codec == CODAG_CODEC_DEFLATE) return !(flags & kInflateWarps) || !InflateJob(d).small();
  return d.out_len >= kWarpBytes && rle_team_takes(a, d) && rle_team_pays(d, (flags & ~kAnyTeam) >> kShiftAt);
}
__global__ void __launch_bounds__(1024) k_classify(BatchArgs a, uint32_t n, uint32_t resident, uint32_t* __restrict__ queue) {
  __shared__ uint32_t long_v2[kShifts];
  __shared__ float small_team;
  __shared__ int small_longest;  // a float's bits, which compare as it does
  if (threadIdx.x < kShifts) long_v2[threadIdx.x] = 0;
  if (threadIdx.x == 0) small_team = small_longest = 0;
  __syncthreads();
  bool any = false, large = false;  // there are files for teams; Deflate files among them that warps do not take
  SmallInflates mine;
#pragma unroll 4
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
    const codag_chunk_desc d = a.descs[i];
    if (d.codec == CODAG_CODEC_DEFLATE) {
      const InflateJob j(d);
      mine.add(j);
      large |= !j.small();
    } else if (wants_team(a, d, 0)) {
      if (d.codec != CODAG_CODEC_RLEV2) any = true;
      else atomicAdd(&long_v2[shifts_below(d.out_len)], 1u);
    }
  }
  if (mine.team > 0) {
    atomicAdd(&small_team, mine.team);
    atomicMax(&small_longest, __float_as_int(mine.longest));
  }
  any = __syncthreads_or(any || large);
  if (threadIdx.x != 0) return;
  mine.team = small_team;
  mine.longest = __int_as_float(small_longest);
  const bool warps = mine.by_warps(resident);
  any |= mine.team > 0 && !warps;
  const uint32_t shift = v2_shift(long_v2, resident);
  for (uint32_t j = shift + 1; j < kShifts; j++) any |= long_v2[j] != 0;
  *queue = (any ? kAnyTeam : 0u) | (warps ? kInflateWarps : 0u) | (shift << kShiftAt);
}

// Entries [0, n) of the order, each taken by the CTA's warps together, an RLE stream that a team cannot take by
// the first alone; MIXED: those for a team, the others are passed over.  False after a timeout; else sh.job is
// what the queue gave after the last entry.
template <bool MIXED>
__device__ __forceinline__ bool team_jobs(const BatchArgs& a, uint64_t n, uint32_t* queue, BatchShared& sh, uint64_t wait_cycles,
                                          uint32_t warp, uint32_t lane, RleRing& rle) {
  InflateTeam& sm = sh.inflate;
  InflateRing in;
  TokenRing tin;
  InflateWin o;
  inflate_rings(in, tin, sm, wait_cycles, warp, lane);
  inflate_window(o, sm, lane);
  if (warp == 5) init_ring_barriers<16>(sh.tb.bar, lane);
  if (threadIdx.x == 0) sh.tb.phase = 0;
  for (;;) {
    if (threadIdx.x == 0) {
      sh.job = atomicAdd(queue, 1u);
      sh.ahead = 0xffffffffu;
      sh.st = CODAG_OK;
      sm.stop = sm.dead = 0;
    }
    __syncthreads();
    const uint32_t job = sh.job, k = MIXED ? job & ((1u << kCountBits) - 1u) : job;
    if (k >= n || (MIXED && !(job & kAnyTeam))) return true;
    const uint32_t i = a.order ? a.order[k] : k;
    const codag_chunk_desc d = a.descs[i];
    if constexpr (MIXED) {
      if (!wants_team(a, d, job)) {  // on to the next entry for a team, if it is among those the threads look at
        constexpr uint32_t kLook = 8;
        uint32_t far = k + 1u + kLook * 32u * kWarps;
        if (far > n) far = static_cast<uint32_t>(n);
#pragma unroll
        for (uint32_t q = 0; q < kLook; q++) {
          const uint32_t e = k + 1u + q * 32u * kWarps + threadIdx.x;
          if (e < far && wants_team(a, a.descs[a.order ? a.order[e] : e], job)) far = e;
        }
        far = __reduce_min_sync(FULL, far);
        if (lane == 0) atomicMin(&sh.ahead, far);
        __syncthreads();
        if (threadIdx.x == 0) atomicMax(queue, (job & ~((1u << kCountBits) - 1u)) | sh.ahead);
        continue;
      }
    }
    if (d.codec != CODAG_CODEC_DEFLATE) {
      uint32_t state = kTeamFallback;
      if (rle_team_takes(a, d) &&
          (d.codec == CODAG_CODEC_RLEV1 || !rlev2_alone(a.comp + d.comp_off, d.comp_len, d.out_len / d.elem_bytes)))
        state = d.codec == CODAG_CODEC_RLEV1 ? rle_team_any<CODAG_CODEC_RLEV1>(sh.v1, sh.tb, a, d, wait_cycles)
                                             : rle_team_any<CODAG_CODEC_RLEV2>(sh.v2, sh.tb, a, d, wait_cycles);
      if (warp == 0) {
        int st = state == kTeamTimeout ? CODAG_ETIMEOUT : state == kTeamShort ? CODAG_ECORRUPT : CODAG_OK;
        if (state == kTeamFallback) {
          fence_proxy_async_smem();
          st = warp_job(a, d, rle, sh.one[0], lane);
        }
        if (lane == 0) {
          if (a.status) a.status[i] = st;
          sh.st = st;
        }
      }
    } else if (!job_in_bounds(a, d)) {
      if (a.status && threadIdx.x == 0) a.status[i] = CODAG_ECORRUPT;
    } else if (warp < 2) {
      in.begin(a.comp + d.comp_off, d.comp_len);
      inflate_scan(in, sm, d.wrapper_bytes, warp, lane);
    } else if (warp < 4) {
      tin.begin(a.comp + d.comp_off, d.comp_len);
      inflate_tokens(tin, sm, warp - 2u, lane);
    } else if (warp == 4) {
      inflate_place(sm, d.out_len, lane);
    } else {
      o.begin(a.out + d.out_off, d.out_len);
      const int st = inflate_copy(sm, o, a.comp + d.comp_off, d.comp_len, lane);
      if (lane == 0) {
        if (a.status) a.status[i] = st;
        sh.st = sm.dead || sm.status == CODAG_ETIMEOUT ? static_cast<int>(CODAG_ETIMEOUT) : st;
      }
    }
    fence_proxy_async_smem();  // the next stream's bytes may come in where this one's tables are
    __syncthreads();
    const bool timed_out = sh.st == CODAG_ETIMEOUT;
    __syncthreads();  // every warp has looked before the next job resets it
    if (timed_out) return false;  // ring state unknown: the CTA stops
  }
}

// Entries [n0, n) of the order, one per warp; MIXED: those not for a team, the first warp beginning with
// `job`, which its CTA has taken already.
template <bool MIXED>
__device__ __forceinline__ void warp_jobs(const BatchArgs& a, uint64_t n0, uint64_t n, uint32_t job, uint32_t* queue, uint32_t warp,
                                          uint32_t lane, RleRing& in, OneWarp& sh) {
  // a list of fewer than the grid's warps, and none for teams: the CTAs share it evenly (600 of 128 KiB: 217 us | 185)
  if (MIXED && !(job & kAnyTeam) && warp * gridDim.x >= n) return;
  bool have = MIXED && warp == 0;
  for (;;) {
    if (!have && lane == 0) job = atomicAdd(queue, 1u);
    have = false;
    job = __shfl_sync(FULL, job, 0);
    uint32_t k = job;
    if (MIXED) {
      k &= (1u << kCountBits) - 1u;
      if (job & kAnyTeam) k -= static_cast<uint32_t>(n);  // the list's second time
    }
    if (k >= n - n0) break;
    const uint32_t i = a.order ? a.order[n0 + k] : static_cast<uint32_t>(n0) + k;
    const codag_chunk_desc& d = a.descs[i];
    if (MIXED && (job & kAnyTeam) && wants_team(a, d, job)) continue;
    const int st = warp_job(a, d, in, sh, lane);
    if (a.status && lane == 0) a.status[i] = st;
    if (st == CODAG_ETIMEOUT) break;  // ring state unknown: this warp stops pulling work
  }
}

// Persistent grid, three CTAs per SM.  The first n_team entries of the order are taken by CTAs
// (queue[0]), longest first; the others, a plan's short RLE files, by single warps (queue[1]), which
// fills the SMs while the last of the CTAs' streams are decoded.  MIXED: the list is in no such order, and
// n_team is n.
template <bool MIXED>
__global__ void __launch_bounds__(32 * kWarps, 3)
    k_batch(BatchArgs a, uint64_t n, uint64_t n_team, uint32_t* __restrict__ queue, uint64_t wait_cycles) {
  extern __shared__ __align__(128) uint8_t smem[];
  BatchShared& sh = *reinterpret_cast<BatchShared*>(smem);
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  RleRing rle;
  rle_ring(rle, sh.one[warp], sh.bar[warp], wait_cycles, lane);
  if (n_team && !team_jobs<MIXED>(a, n_team, queue, sh, wait_cycles, warp, lane, rle)) return;
  if (MIXED) warp_jobs<true>(a, 0, n, sh.job, queue, warp, lane, rle, sh.one[warp]);
  else if (n_team < n) warp_jobs<false>(a, n_team, n, 0, queue + 1, warp, lane, rle, sh.one[warp]);
}

// A plan without files for teams: as many warps as an SM has registers for.
constexpr uint32_t kFew = 2, kFewCtas = 12;
__global__ void __launch_bounds__(32 * kFew, kFewCtas)
    k_batch_warps(BatchArgs a, uint64_t n, uint32_t* __restrict__ queue, uint64_t wait_cycles) {
  __shared__ OneWarp one[kFew];
  __shared__ uint64_t bar[kFew][4];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  RleRing rle;
  rle_ring(rle, one[warp], bar[warp], wait_cycles, lane);
  warp_jobs<false>(a, 0, n, 0, queue, warp, lane, rle, one[warp]);
}

}  // namespace

struct codag_plan {
  uint64_t n = 0;
  uint64_t n_team = 0;  // leading entries of the order, taken by CTAs
  codag_chunk_desc* d_descs = nullptr;
  uint32_t* d_order = nullptr;
  uint32_t* d_queue = nullptr;
  int grid = 0, mixed_grid = 0;
  // captured graph and the arguments it was captured with
  cudaGraphExec_t exec = nullptr;
  const void* g_comp = nullptr;
  const void* g_out = nullptr;
  const void* g_status = nullptr;
  uint64_t g_comp_bytes = 0, g_out_bytes = 0;
};

namespace {

// CTAs of the persistent grid on the current device: as many as are resident at once
codag_status batch_grid_cap(int* cap) {
  if (allow_smem(k_batch<false>, sizeof(BatchShared)) != cudaSuccess || allow_smem(k_batch<true>, sizeof(BatchShared)) != cudaSuccess)
    return CODAG_ECUDA;
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return CODAG_ECUDA;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch<false>, 32 * kWarps, sizeof(BatchShared)) != cudaSuccess)
    return CODAG_ECUDA;
  *cap = sms * std::max(per_sm, 1);
  return CODAG_OK;
}

void batch_enqueue(const BatchArgs& a, uint64_t n, uint64_t n_team, uint32_t* queue, int grid, cudaStream_t s) {
  cudaMemsetAsync(queue, 0, (n_team < n ? 2 : 1) * sizeof(uint32_t), s);
  if (n_team == 0) k_batch_warps<<<grid, 32 * kFew, 0, s>>>(a, n, queue, wait_of());
  else k_batch<false><<<grid, 32 * kWarps, sizeof(BatchShared), s>>>(a, n, n_team, queue, wait_of());
}
void mixed_enqueue(const BatchArgs& a, uint64_t n, uint32_t* queue, uint64_t resident, cudaStream_t s) {
  const int grid = static_cast<int>(std::min(n, resident));
  // with a CTA for each there is nothing to find out (200 Deflate files of 1 KiB: 65 us with the small kernel, 58)
  if (n <= resident || n > kMaxMixed) return batch_enqueue(a, n, n, queue, grid, s);
  k_classify<<<1, n < 1024 ? static_cast<unsigned>((n + 31) / 32 * 32) : 1024u, 0, s>>>(a, static_cast<uint32_t>(n), static_cast<uint32_t>(resident), queue);
  k_batch<true><<<grid, 32 * kWarps, sizeof(BatchShared), s>>>(a, n, n, queue, wait_of());
}
// CTAs decode RLE files whose output is element aligned; a plan checks the offsets, so the base has to be, too
void plan_enqueue(const codag_plan& p, const BatchArgs& a, cudaStream_t s) {
  if (reinterpret_cast<uintptr_t>(a.out) % 8) mixed_enqueue(a, p.n, p.d_queue, static_cast<uint64_t>(p.mixed_grid), s);
  else batch_enqueue(a, p.n, p.n_team, p.d_queue, p.grid, s);
}

// Work estimate that orders the queue: a Deflate stream takes some 3 us per KiB of output, an RLE
// stream on a CTA a third to a sixth of that.
uint64_t chunk_cost(const codag_chunk_desc& d) {
  return d.codec == CODAG_CODEC_DEFLATE ? 8ull * d.comp_len + d.out_len : static_cast<uint64_t>(d.comp_len) + d.out_len / 4;
}

// CTAs of the grid.  One stream alone on an SM is decoded 2.5 times as fast as three side by side, so
// when the longest takes more than an even share of the work on two CTAs per SM, no more are started
// (2000 files of 4 KiB to 1 MiB: 3.2 ms | 3.7; 2048 Deflate files of 128 KiB: 2.9 | 2.3).
uint64_t grid_cap(uint64_t resident, uint64_t longest, uint64_t total) {
  const uint64_t two = std::max<uint64_t>(resident * 2 / 3, 1);
  return longest > total / two ? two : resident;
}

bool valid_shape(const codag_tune& t) {
  return valid_warps(t.warps_per_cta) && valid_slots(t.ring_slots) && valid_lut(t.lut_bits);
}

}  // namespace

extern "C" codag_status codag_batch_plan(const codag_chunk_desc* h_descs, uint64_t n, const codag_tune* tune,
                                         codag_plan** plan) {
  if (!h_descs || !plan || n == 0 || n > 0xffffffffull) return CODAG_EINVAL;
  if (tune) {
    if (!valid_shape(*tune)) return CODAG_EINVAL;
    if (tune->cta_per_chunk < 0 || tune->cta_per_chunk > 4 || (tune->cta_per_chunk && (tune->warps_per_cta & 1)))
      return CODAG_EINVAL;
    if (tune->table_global != 0 && tune->table_global != 1) return CODAG_EINVAL;
  }
  for (uint64_t i = 0; i < n; i++) {
    const codag_chunk_desc& d = h_descs[i];
    if (d.codec > CODAG_CODEC_DEFLATE) return CODAG_EINVAL;
    if (d.codec != CODAG_CODEC_DEFLATE && (!valid_elem(d.elem_bytes) || d.out_len % d.elem_bytes)) return CODAG_EINVAL;
  }
  codag_plan* p = new (std::nothrow) codag_plan();
  if (!p) return CODAG_ENOMEM;
  p->n = n;
  std::vector<uint32_t> order(n);
  for (uint64_t i = 0; i < n; i++) order[i] = static_cast<uint32_t>(i);
  int cap = 0;
  const codag_status st = batch_grid_cap(&cap);
  if (st != CODAG_OK) {
    codag_batch_destroy(p);
    return st;
  }
  uint32_t long_v2[kShifts] = {};
  for (uint64_t i = 0; i < n; i++)
    if (h_descs[i].codec == CODAG_CODEC_RLEV2 && rle_team_pays(h_descs[i], 0)) long_v2[shifts_below(h_descs[i].out_len)]++;
  const uint32_t shift = v2_shift(long_v2, static_cast<uint64_t>(cap));
  SmallInflates small;
  for (uint64_t i = 0; i < n; i++)
    if (h_descs[i].codec == CODAG_CODEC_DEFLATE) small.add(InflateJob(h_descs[i]));
  const bool inflate_warps = small.by_warps(static_cast<uint64_t>(cap));
  const auto team = [&](uint32_t i) {
    const codag_chunk_desc& d = h_descs[i];
    if (d.codec == CODAG_CODEC_DEFLATE) return !inflate_warps || !InflateJob(d).small();
    return (rle_team_pays(d, shift) && d.out_off % d.elem_bytes == 0);
  };
  uint64_t longest = 0, total = 0;
  for (uint64_t i = 0; i < n; i++) {
    const uint64_t cost = chunk_cost(h_descs[i]);
    longest = std::max(longest, cost);
    total += cost;
  }
  std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) {
    if (team(a) != team(b)) return team(a);
    return chunk_cost(h_descs[a]) > chunk_cost(h_descs[b]);
  });
  while (p->n_team < n && team(order[p->n_team])) p->n_team++;
  if (cudaMalloc(&p->d_descs, n * sizeof(codag_chunk_desc)) != cudaSuccess ||
      cudaMalloc(&p->d_order, n * sizeof(uint32_t)) != cudaSuccess ||
      cudaMalloc(&p->d_queue, 2 * sizeof(uint32_t)) != cudaSuccess ||
      cudaMemcpy(p->d_descs, h_descs, n * sizeof(codag_chunk_desc), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(p->d_order, order.data(), n * sizeof(uint32_t), cudaMemcpyHostToDevice) != cudaSuccess) {
    codag_batch_destroy(p);
    return CODAG_ECUDA;
  }
  const uint64_t need = p->n_team + (n - p->n_team + kWarps - 1) / kWarps;
  p->grid = static_cast<int>(std::min<uint64_t>(need, grid_cap(static_cast<uint64_t>(cap), longest, total)));
  p->mixed_grid = cap;
  if (p->n_team == 0) p->grid = static_cast<int>(std::min<uint64_t>((n + kFew - 1) / kFew, static_cast<uint64_t>(cap) / 3 * kFewCtas));
  *plan = p;
  return CODAG_OK;
}

extern "C" codag_status codag_batch_run(codag_plan* p, const uint8_t* d_comp, uint64_t comp_bytes, uint8_t* d_out,
                                        uint64_t out_bytes, int32_t* d_status, int use_graph, codag_stream_t stream) {
  if (!p || !d_comp || !d_out) return CODAG_EINVAL;
  clear_stale_error();
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const BatchArgs args{p->d_descs, p->d_order, d_comp, comp_bytes, d_out, out_bytes, d_status};
  if (!use_graph) {
    plan_enqueue(*p, args, s);
    return finish_launch();
  }
  const bool same = p->exec && p->g_comp == d_comp && p->g_out == d_out && p->g_status == d_status &&
                    p->g_comp_bytes == comp_bytes && p->g_out_bytes == out_bytes;
  if (!same) {
    if (p->exec) {
      cudaGraphExecDestroy(p->exec);
      p->exec = nullptr;
    }
    cudaStream_t cap;
    if (cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking) != cudaSuccess) return CODAG_ECUDA;
    cudaGraph_t g = nullptr;
    cudaError_t err = cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
    if (err == cudaSuccess) {
      plan_enqueue(*p, args, cap);
      err = cudaStreamEndCapture(cap, &g);
    }
    if (err == cudaSuccess) err = cudaGraphInstantiate(&p->exec, g, 0);
    if (g) cudaGraphDestroy(g);
    cudaStreamDestroy(cap);
    if (err != cudaSuccess) {
      p->exec = nullptr;
      cudaGetLastError();
      return CODAG_ECUDA;
    }
    p->g_comp = d_comp;
    p->g_out = d_out;
    p->g_status = d_status;
    p->g_comp_bytes = comp_bytes;
    p->g_out_bytes = out_bytes;
  }
  return cudaGraphLaunch(p->exec, s) == cudaSuccess ? CODAG_OK : CODAG_ECUDA;
}

extern "C" codag_status codag_batch_destroy(codag_plan* p) {
  if (!p) return CODAG_EINVAL;
  if (p->exec) cudaGraphExecDestroy(p->exec);
  if (p->d_descs) cudaFree(p->d_descs);
  if (p->d_order) cudaFree(p->d_order);
  if (p->d_queue) cudaFree(p->d_queue);
  delete p;
  return CODAG_OK;
}

// ---------------------------------------------------------------------------------------
// launches over caller-owned descriptor lists (continuous batching)
// ---------------------------------------------------------------------------------------
namespace {
std::mutex g_cap_mu;
std::vector<std::pair<int, int>> g_caps;  // (device, CTAs of the persistent grid)

codag_status cached_grid_cap(int* cap) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return CODAG_ECUDA;
  std::lock_guard<std::mutex> g(g_cap_mu);
  for (const auto& c : g_caps)
    if (c.first == dev) {
      *cap = c.second;
      return CODAG_OK;
    }
  const codag_status st = batch_grid_cap(cap);
  if (st == CODAG_OK) g_caps.push_back({dev, *cap});
  return st;
}
}  // namespace

extern "C" codag_status codag_batch_launch(const codag_chunk_desc* d_descs, const uint32_t* d_order, uint64_t n,
                                           uint32_t* d_queue, const codag_tune* tune, const uint8_t* d_comp,
                                           uint64_t comp_bytes, uint8_t* d_out, uint64_t out_bytes,
                                           int32_t* d_status, codag_stream_t stream) {
  if (!d_descs || !d_queue || !d_comp || !d_out || n > 0xffffffffull) return CODAG_EINVAL;
  if (n == 0) return CODAG_OK;
  clear_stale_error();
  if (tune && (!valid_shape(*tune) || tune->table_global)) return CODAG_EINVAL;
  int cap = 0;
  const codag_status st = cached_grid_cap(&cap);
  if (st != CODAG_OK) return st;
  const BatchArgs args{d_descs, d_order, d_comp, comp_bytes, d_out, out_bytes, d_status};
  mixed_enqueue(args, n, d_queue, static_cast<uint64_t>(cap), reinterpret_cast<cudaStream_t>(stream));
  return finish_launch();
}
