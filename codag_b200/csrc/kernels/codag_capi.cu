// RLE decoders: per-file kernels and entry points (include/codag.h), and the process-wide
// settings of the library.
//
// Plain per-file launches: one warp per chunk, `warps_per_cta` chunks per CTA, each warp
// with its own slice of dynamic shared memory (TMA input ring [+ output ring]).
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <type_traits>
#include <utility>
#include <vector>

#include "capi_common.cuh"
#include "decode_rle_team.cuh"
#include "walk_rle.cuh"

using namespace codag_dev;
using namespace codag_capi;

namespace {

// ---------------------------------------------------------------------------------------
// per-warp shared memory layouts
// ---------------------------------------------------------------------------------------

using RleOut = OutRing<12, 10, true>;  // 4 KiB ring, 1 KiB drains by TMA bulk stores
template <int NSLOT>
struct RleLayout {
  static constexpr uint32_t kIn = 0;
  static constexpr uint32_t kOut = kIn + align_up(InRing<NSLOT>::kAlloc, 128);
  static constexpr uint32_t kBar = kOut + RleOut::kBytes;
  static constexpr uint32_t kPerWarp = align_up(kBar + NSLOT * 8, 128);
};

// RLE with DirectOut: no output ring
template <int NSLOT>
struct RleDirectLayout {
  static constexpr uint32_t kIn = 0;
  static constexpr uint32_t kBar = kIn + InRing<NSLOT>::kAlloc;
  static constexpr uint32_t kPerWarp = align_up(kBar + NSLOT * 8, 128);
};

// ---------------------------------------------------------------------------------------
// plain kernels: chunk = blockIdx.x * warps + warp
// ---------------------------------------------------------------------------------------
// header walk, one thread per chunk; descriptors and counts go to the workspace
template <int CODEC>
__global__ void __launch_bounds__(128) k_rle_walk(const uint8_t* __restrict__ comp, uint64_t comp_bytes,
                                                  const uint64_t* __restrict__ blk_off,
                                                  const uint64_t* __restrict__ col_len, uint64_t n_chunks,
                                                  uint32_t cap, uint32_t* __restrict__ counts,
                                                  RleDesc* __restrict__ descs) {
  const uint64_t chunk = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (chunk >= n_chunks) return;
  const uint64_t off = blk_off[chunk], len = col_len[chunk];
  uint32_t k = kWalkFallback;
  if (stream_in_bounds(off, len, comp_bytes)) {
    const GStream g{comp + off, static_cast<uint32_t>(len), comp, comp + comp_bytes};
    RleDesc* d = descs + chunk * kDescPerChunk;
    k = CODEC == CODAG_CODEC_RLEV1 ? walk_rlev1(g, cap, d) : walk_rlev2(g, cap, d);
  }
  counts[chunk] = k;
}

template <int NSLOT, int CODEC, int E, bool DIRECT>
__global__ void __launch_bounds__(256) k_rle_plain(const uint8_t* __restrict__ comp, uint64_t comp_bytes,
                                                   const uint64_t* __restrict__ blk_off,
                                                   const uint64_t* __restrict__ col_len, uint64_t n_chunks,
                                                   uint64_t chunk_bytes, uint8_t* __restrict__ out,
                                                   uint64_t out_bytes, int32_t* __restrict__ status,
                                                   uint64_t wait_cycles, const uint32_t* __restrict__ counts,
                                                   const RleDesc* __restrict__ descs) {
  extern __shared__ __align__(128) uint8_t smem[];
  using L = std::conditional_t<DIRECT, RleDirectLayout<NSLOT>, RleLayout<NSLOT>>;
  using OUT = std::conditional_t<DIRECT, DirectOut, RleOut>;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint64_t chunk = static_cast<uint64_t>(blockIdx.x) * (blockDim.x >> 5) + warp;
  if (chunk >= n_chunks) return;
  uint8_t* base = smem + warp * L::kPerWarp;
  InRing<NSLOT> in;
  in.buf = base + L::kIn;
  in.sbuf = smem_u32(in.buf);
  in.bar = reinterpret_cast<uint64_t*>(base + L::kBar);
  in.phase = 0;
  in.wait_cycles = wait_cycles;
  in.lane = lane;
  OUT o;
  if constexpr (!DIRECT) {
    o.buf = base + L::kOut;
    o.sbuf = smem_u32(o.buf);
  }
  o.lane = lane;
  init_ring_barriers<NSLOT>(in.bar, lane);

  const uint64_t off = blk_off[chunk], len = col_len[chunk];
  const uint64_t cbase = chunk * chunk_bytes;
  int st;
  if (!stream_in_bounds(off, len, comp_bytes)) {
    st = CODAG_ECORRUPT;
  } else {
    in.begin(comp + off, static_cast<uint32_t>(len));
    o.begin(out + cbase, store_bytes(cbase, chunk_bytes, out_bytes));
    const uint32_t cap = static_cast<uint32_t>(chunk_bytes / E);
    const uint32_t nd = counts ? counts[chunk] : kWalkFallback;
    if (nd != kWalkFallback) {
      const RleDesc* d = descs + chunk * kDescPerChunk;
      st = CODEC == CODAG_CODEC_RLEV1 ? expand_rlev1<NSLOT, E>(in, o, d, nd) : expand_rlev2<NSLOT, E>(in, o, d, nd);
    } else {
      st = CODEC == CODAG_CODEC_RLEV1 ? decode_rlev1_chunk<NSLOT, E>(in, o, cap) : decode_rlev2_chunk<NSLOT, E>(in, o, cap);
    }
  }
  if (status && lane == 0) status[chunk] = st;
}

// ---------------------------------------------------------------------------------------
// one CTA per chunk (decode_rle_team.cuh), values straight to global memory
// ---------------------------------------------------------------------------------------
template <int CODEC>
constexpr uint32_t kTeamWarpsOf = CODEC == CODAG_CODEC_RLEV1 ? 8 : 16;
template <int CODEC>
struct TeamShared {
  std::conditional_t<CODEC == CODAG_CODEC_RLEV1, TeamV1, TeamV2<6>> team;
  TeamBars tb;
  uint64_t bar4[4];
};

// The chunk by one warp, from the start, through the first part of the team's ring.
template <int CODEC, int E>
__device__ __noinline__ int decode_alone(uint8_t* ring, uint64_t* bar, const uint8_t* src, uint32_t len, uint8_t* dst, uint32_t store,
                                         uint32_t cap, uint64_t wait_cycles, uint32_t lane) {
  DirectOut o;
  o.lane = lane;
  o.begin(dst, store);
  InRing<4> one;
  one.buf = ring;
  one.sbuf = smem_u32(ring);
  one.bar = bar;
  one.phase = 0;
  one.wait_cycles = wait_cycles;
  one.lane = lane;
  init_ring_barriers<4>(one.bar, lane);
  fence_proxy_async_smem();
  one.begin(src, len);
  return CODEC == CODAG_CODEC_RLEV1 ? decode_rlev1_chunk<4, E>(one, o, cap) : decode_rlev2_chunk<4, E>(one, o, cap);
}

// RLE v2: two CTAs a SM, as the compiler spills to fit three otherwise (3 MB of 16-bit values 179 us | 164)
template <int CODEC, int E>
__global__ void __launch_bounds__(32 * kTeamWarpsOf<CODEC>, CODEC == CODAG_CODEC_RLEV2 ? 2 : 6)
    k_rle_team(const uint8_t* __restrict__ comp, uint64_t comp_bytes, const uint64_t* __restrict__ blk_off,
               const uint64_t* __restrict__ col_len, uint64_t chunk_bytes, uint8_t* __restrict__ out, uint64_t out_bytes,
               int32_t* __restrict__ status, uint64_t wait_cycles) {
  extern __shared__ __align__(128) uint8_t smem[];
  TeamShared<CODEC>& sh = *reinterpret_cast<TeamShared<CODEC>*>(smem);
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint64_t chunk = blockIdx.x;
  const uint64_t off = blk_off[chunk], len = col_len[chunk];
  const uint64_t cbase = chunk * chunk_bytes;
  const uint32_t cap = static_cast<uint32_t>(chunk_bytes / E), store = store_bytes(cbase, chunk_bytes, out_bytes);
  if (!stream_in_bounds(off, len, comp_bytes)) {
    if (status && threadIdx.x == 0) status[chunk] = CODAG_ECORRUPT;
    return;
  }
  uint32_t state = kTeamFallback;
  if (CODEC == CODAG_CODEC_RLEV1 || !rlev2_alone(comp + off, static_cast<uint32_t>(len), cap)) {
    if (warp == 1) init_ring_barriers<16>(sh.tb.bar, lane);
    if (threadIdx.x == 0) sh.tb.phase = 0;
    __syncthreads();
    state = rle_team<CODEC, E, kTeamWarpsOf<CODEC>>(sh.team, sh.tb, comp + off, static_cast<uint32_t>(len), out + cbase, store,
                                                    cap, wait_cycles);
  }
  if (warp != 0) return;
  int st = state == kTeamTimeout ? CODAG_ETIMEOUT : state == kTeamShort ? CODAG_ECORRUPT : CODAG_OK;
  if (state == kTeamFallback)
    st = decode_alone<CODEC, E>(sh.team.ring, sh.bar4, comp + off, static_cast<uint32_t>(len), out + cbase, store, cap, wait_cycles,
                                lane);
  if (status && lane == 0) status[chunk] = st;
}

// A wait that no copy ever completes: exercises the bounded-wait path of InRing.
__global__ void k_selftest_timeout(int32_t* status, uint64_t wait_cycles) {
  __shared__ __align__(128) uint8_t buf[InRing<1>::kAlloc];
  __shared__ uint64_t bar[1];
  const uint32_t lane = threadIdx.x & 31u;
  InRing<1> in;
  in.buf = buf;
  in.sbuf = smem_u32(buf);
  in.bar = bar;
  in.phase = 0;
  in.wait_cycles = wait_cycles;
  in.lane = lane;
  init_ring_barriers<1>(bar, lane);
  if (lane == 0) mbar_arrive_expect_tx(&bar[0], 16);  // 16 bytes are expected, none is sent
  __syncwarp();
  const bool ok = in.wait_slot(0);
  if (lane == 0) *status = ok ? CODAG_OK : CODAG_ETIMEOUT;
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
std::mutex g_mu;
codag_tune g_tune[3] = {{8, 4, 10, 0, 0}, {8, 4, 10, 0, 0}, {2, 2, 9, 0, 0}};
uint64_t g_wait_cycles = 2000000000ull;  // about one second at 2 GHz

codag_tune tune_of(int codec) {
  std::lock_guard<std::mutex> g(g_mu);
  return g_tune[codec];
}
}  // namespace

uint64_t codag_capi::wait_of() {
  std::lock_guard<std::mutex> g(g_mu);
  return g_wait_cycles;
}

cudaError_t codag_capi::allow_smem_of(const void* kernel, uint32_t bytes) {
  static std::mutex mu;
  static std::vector<std::pair<std::pair<const void*, int>, uint32_t>> set;  // (kernel, device) -> limit set
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  std::lock_guard<std::mutex> g(mu);
  for (auto& e : set)
    if (e.first.first == kernel && e.first.second == dev) {
      if (e.second >= bytes) return cudaSuccess;
      err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
      if (err == cudaSuccess) e.second = bytes;
      return err;
    }
  err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
  if (err == cudaSuccess) set.push_back({{kernel, dev}, bytes});
  return err;
}

namespace {

// workspace of the two-pass RLE path: per-chunk descriptor counts, then descriptor tables
constexpr uint64_t rle_ws_counts_bytes(uint64_t n) { return (n * 4 + 255) / 256 * 256; }
constexpr uint64_t rle_ws_bytes(uint64_t n) { return rle_ws_counts_bytes(n) + n * kDescPerChunk * sizeof(RleDesc); }

constexpr uint64_t kSms = 148;

template <int NSLOT, int CODEC, int E, bool DIRECT>
codag_status launch_rle_out(const codag_tune& t, const uint8_t* comp, uint64_t comp_bytes, const uint64_t* blk_off,
                            const uint64_t* col_len, uint64_t n, uint64_t chunk_bytes, uint8_t* out,
                            uint64_t out_bytes, int32_t* status, void* ws, uint64_t ws_bytes, cudaStream_t s) {
  using L = std::conditional_t<DIRECT, RleDirectLayout<NSLOT>, RleLayout<NSLOT>>;
  // With more chunks than warps are resident (32 per SM), CTAs of four warps in the place of the default's eight: a slot is
  // taken again as soon as its four are done (RLE v2, 1 GiB of 64-bit values 438 us with eight, 428 with four, 700 MB
  // of 32-bit values 615 | 595; 256 MiB, all resident at once, 190 | 191; not measured with a workspace or the ring).
  const int warps = DIRECT && !ws && n > 32 * kSms && t.warps_per_cta == 8 ? 4 : t.warps_per_cta;
  const uint32_t smem = L::kPerWarp * warps;
  auto kern = k_rle_plain<NSLOT, CODEC, E, DIRECT>;
  if (allow_smem(kern, smem) != cudaSuccess) return CODAG_ECUDA;
  const uint64_t grid = (n + warps - 1) / warps;
  if (grid > 0x7fffffffull) return CODAG_EINVAL;
  uint32_t* counts = nullptr;
  RleDesc* descs = nullptr;
  if (ws && ws_bytes >= rle_ws_bytes(n) && (reinterpret_cast<uintptr_t>(ws) & 255) == 0) {
    counts = static_cast<uint32_t*>(ws);
    descs = reinterpret_cast<RleDesc*>(static_cast<uint8_t*>(ws) + rle_ws_counts_bytes(n));
    k_rle_walk<CODEC><<<static_cast<unsigned>((n + 127) / 128), 128, 0, s>>>(
        comp, comp_bytes, blk_off, col_len, n, static_cast<uint32_t>(chunk_bytes / E), counts, descs);
  }
  kern<<<static_cast<unsigned>(grid), 32 * warps, smem, s>>>(comp, comp_bytes, blk_off, col_len, n, chunk_bytes, out, out_bytes,
                                                             status, wait_of(), counts, descs);
  return finish_launch();
}

template <int CODEC, int E>
codag_status launch_rle_team(const uint8_t* comp, uint64_t comp_bytes, const uint64_t* blk_off, const uint64_t* col_len,
                             uint64_t n, uint64_t chunk_bytes, uint8_t* out, uint64_t out_bytes, int32_t* status,
                             cudaStream_t s) {
  constexpr uint32_t smem = sizeof(TeamShared<CODEC>);
  auto kern = k_rle_team<CODEC, E>;
  if (allow_smem(kern, smem) != cudaSuccess) return CODAG_ECUDA;
  if (n > 0x7fffffffull) return CODAG_EINVAL;
  kern<<<static_cast<unsigned>(n), 32 * kTeamWarpsOf<CODEC>, smem, s>>>(comp, comp_bytes, blk_off, col_len, chunk_bytes, out,
                                                                      out_bytes, status, wait_of());
  return finish_launch();
}

// Whether a team for each chunk is faster than a warp for each (measured, us, team | warp).
//   RLE v1: up to about two chunks for each resident CTA, always (700 chunks: 17 | 20 at 6 bytes of stream each, 168 |
//   715 at 152 KiB).  With more, a chunk also costs 2 us of a CTA's place, which the length of the streams has to
//   earn back: 64-bit values, 2048 chunks: 25 | 20 at 6 bytes, 31 | 27 at 780, 49 | 51 at 3000, 187 | 272 at
//   24 KiB; 8192 chunks: 51 | 21, 76 | 45, 144 | 110, 374 | 373 at 12 KiB, 458 | 704 at 38 KiB; 8 and 32 bits the
//   same within a fifth.  The mean stream is taken from comp_bytes (too
//   long for a part of a file, too short where chunks share a stream).
//   RLE v2 (the look-ahead reads every byte as a header, which pays while SMs have room for it): 64-bit
//   values: 32 chunks 80 | 138, 400 146 | 157, 640 204 | 175; 16 bits: 32 168 | 424, 400 370 | 479,
//   640 527 | 484; 8 bits: 640 808 | 825, 1280 1389 | 884.  Not for short streams (64-bit values, 8 chunks: 20 | 17 at
//   144 bytes), nor where chunks are small and their streams are those that a team leaves to one of its warps
//   (64-bit values, 32 chunks of 2 KiB: 19 | 16).
template <int CODEC>
bool team_pays(uint64_t n, uint64_t comp_bytes, uint64_t values) {
  const uint64_t mean = comp_bytes / n;
  if (CODEC == CODAG_CODEC_RLEV2) return n <= 3 * kSms && mean > kTeamMinBytes && (values > 1024 || mean <= 2 * values);
  constexpr uint64_t kFree = 900, kAll = 8900;
  return n <= kFree || mean * 4 >= 5 * ((n < kAll ? n : kAll) - kFree);
}

// Values go straight to global memory when the output is element aligned (DirectOut),
// through the shared-memory ring otherwise; with cta_per_chunk (and no workspace) a whole
// CTA decodes each chunk.
template <int NSLOT, int CODEC, int E>
codag_status launch_rle(const codag_tune& t, const uint8_t* comp, uint64_t comp_bytes, const uint64_t* blk_off,
                        const uint64_t* col_len, uint64_t n, uint64_t chunk_bytes, uint8_t* out, uint64_t out_bytes,
                        int32_t* status, void* ws, uint64_t ws_bytes, cudaStream_t s) {
  // direct stores write whole elements: the output and out_bytes must be element aligned
  const bool direct = (reinterpret_cast<uintptr_t>(out) % E) == 0 && out_bytes % E == 0;
  if (direct && !ws && (t.cta_per_chunk || team_pays<CODEC>(n, comp_bytes, chunk_bytes / E)))
    return launch_rle_team<CODEC, E>(comp, comp_bytes, blk_off, col_len, n, chunk_bytes, out, out_bytes, status, s);
  if (direct)
    return launch_rle_out<NSLOT, CODEC, E, true>(t, comp, comp_bytes, blk_off, col_len, n, chunk_bytes, out,
                                                 out_bytes, status, ws, ws_bytes, s);
  return launch_rle_out<NSLOT, CODEC, E, false>(t, comp, comp_bytes, blk_off, col_len, n, chunk_bytes, out, out_bytes,
                                                status, ws, ws_bytes, s);
}

template <int NSLOT, int CODEC>
codag_status launch_rle_e(const codag_tune& t, const uint8_t* comp, uint64_t comp_bytes, const uint64_t* blk_off,
                          const uint64_t* col_len, uint64_t n, uint64_t chunk_bytes, int e, uint8_t* out,
                          uint64_t out_bytes, int32_t* status, void* ws, uint64_t wsb, cudaStream_t s) {
  switch (e) {
    case 8: return launch_rle<NSLOT, CODEC, 8>(t, comp, comp_bytes, blk_off, col_len, n, chunk_bytes, out, out_bytes, status, ws, wsb, s);
    case 4: return launch_rle<NSLOT, CODEC, 4>(t, comp, comp_bytes, blk_off, col_len, n, chunk_bytes, out, out_bytes, status, ws, wsb, s);
    case 2: return launch_rle<NSLOT, CODEC, 2>(t, comp, comp_bytes, blk_off, col_len, n, chunk_bytes, out, out_bytes, status, ws, wsb, s);
    default: return launch_rle<NSLOT, CODEC, 1>(t, comp, comp_bytes, blk_off, col_len, n, chunk_bytes, out, out_bytes, status, ws, wsb, s);
  }
}

template <int CODEC>
codag_status dispatch_rle(const uint8_t* comp, uint64_t comp_bytes, const uint64_t* blk_off, const uint64_t* col_len,
                          uint64_t n, uint64_t chunk_bytes, int e, uint8_t* out, uint64_t out_bytes, int32_t* status,
                          void* ws, uint64_t wsb, cudaStream_t s) {
  if (!comp || !blk_off || !col_len || (!out && out_bytes) || !valid_elem(e) || chunk_bytes == 0 ||
      chunk_bytes % static_cast<uint64_t>(e) || chunk_bytes >= (1ull << 31))
    return CODAG_EINVAL;
  if (n == 0) return CODAG_OK;
  clear_stale_error();
  const codag_tune t = tune_of(CODEC);
  if (t.ring_slots == 4)
    return launch_rle_e<4, CODEC>(t, comp, comp_bytes, blk_off, col_len, n, chunk_bytes, e, out, out_bytes, status, ws, wsb, s);
  return launch_rle_e<8, CODEC>(t, comp, comp_bytes, blk_off, col_len, n, chunk_bytes, e, out, out_bytes, status, ws, wsb, s);
}

}  // namespace

// ---------------------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------------------
extern "C" uint64_t codag_workspace_bytes(int codec, uint64_t n_chunks) {
  return (codec == CODAG_CODEC_RLEV1 || codec == CODAG_CODEC_RLEV2) ? rle_ws_bytes(n_chunks) : 0;
}

extern "C" codag_status codag_decompress_rlev1(const uint8_t* d_comp, uint64_t comp_bytes, const uint64_t* d_blk_off,
                                               const uint64_t* d_col_len, uint64_t n_chunks, uint64_t chunk_bytes,
                                               int elem_bytes, uint8_t* d_out, uint64_t out_bytes,
                                               int32_t* d_chunk_status, void* d_workspace, uint64_t workspace_bytes,
                                               codag_stream_t stream) {
  return dispatch_rle<CODAG_CODEC_RLEV1>(d_comp, comp_bytes, d_blk_off, d_col_len, n_chunks, chunk_bytes, elem_bytes,
                                         d_out, out_bytes, d_chunk_status, d_workspace, workspace_bytes,
                                         reinterpret_cast<cudaStream_t>(stream));
}

extern "C" codag_status codag_decompress_rlev2(const uint8_t* d_comp, uint64_t comp_bytes, const uint64_t* d_blk_off,
                                               const uint64_t* d_col_len, uint64_t n_chunks, uint64_t chunk_bytes,
                                               int elem_bytes, uint8_t* d_out, uint64_t out_bytes,
                                               int32_t* d_chunk_status, void* d_workspace, uint64_t workspace_bytes,
                                               codag_stream_t stream) {
  return dispatch_rle<CODAG_CODEC_RLEV2>(d_comp, comp_bytes, d_blk_off, d_col_len, n_chunks, chunk_bytes, elem_bytes,
                                         d_out, out_bytes, d_chunk_status, d_workspace, workspace_bytes,
                                         reinterpret_cast<cudaStream_t>(stream));
}

// ---------------------------------------------------------------------------------------
// Two-pass RLE v2 decode for callers that cannot allocate device memory.
//
// The scratch is a fixed array in the module's device memory, sized for
// CODAG_NOALLOC_MAX_CHUNKS chunks; every device that loads this library holds it until the
// process exits.  In host code `g_noalloc_ws` only names a host-side shadow, so the device
// address is looked up once per device with cudaGetSymbolAddress (on the first call made
// with that device current) and passed to the kernels.  All calls share the array: the
// header walk rewrites the count of every chunk it is given before the expansion reads it,
// so no clearing is needed, and calls that overlap on the GPU race on the array.
// ---------------------------------------------------------------------------------------
namespace {
constexpr uint64_t kNoAllocScratchBytes = rle_ws_bytes(CODAG_NOALLOC_MAX_CHUNKS);
__device__ __align__(256) uint8_t g_noalloc_ws[kNoAllocScratchBytes];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mu;
void* g_noalloc_addr[kNoAllocMaxDevices] = {};

codag_status noalloc_scratch(void** addr) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return CODAG_ECUDA;
  if (dev < 0 || dev >= kNoAllocMaxDevices) return CODAG_EINVAL;
  std::lock_guard<std::mutex> g(g_noalloc_mu);
  if (!g_noalloc_addr[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_ws) != cudaSuccess || !p) return CODAG_ECUDA;
    g_noalloc_addr[dev] = p;
  }
  *addr = g_noalloc_addr[dev];
  return CODAG_OK;
}
}  // namespace

extern "C" codag_status codag_decompress_rlev2_noalloc(const uint8_t* d_comp, uint64_t comp_bytes,
                                                       const uint64_t* d_blk_off, const uint64_t* d_col_len,
                                                       uint64_t n_chunks, uint64_t chunk_bytes, int elem_bytes,
                                                       uint8_t* d_out, uint64_t out_bytes, int32_t* d_chunk_status,
                                                       codag_stream_t stream) {
  if (!d_comp || !d_blk_off || !d_col_len || (!d_out && out_bytes) || !valid_elem(elem_bytes) || chunk_bytes == 0 ||
      chunk_bytes % static_cast<uint64_t>(elem_bytes) || chunk_bytes >= (1ull << 31))
    return CODAG_EINVAL;  // the checks of dispatch_rle, made before the capacity check
  if (n_chunks > CODAG_NOALLOC_MAX_CHUNKS) return CODAG_ELIMIT;
  if (n_chunks == 0) return CODAG_OK;
  void* ws = nullptr;
  const codag_status st = noalloc_scratch(&ws);
  if (st != CODAG_OK) return st;
  // The two-pass launch takes a workspace only when it is large and 256-byte aligned enough
  // (launch_rle_out); both hold by construction, and if either did not, this call reports it
  // instead of quietly decoding in one pass.
  if ((reinterpret_cast<uintptr_t>(ws) & 255u) != 0 || kNoAllocScratchBytes < rle_ws_bytes(n_chunks)) return CODAG_ECUDA;
  return dispatch_rle<CODAG_CODEC_RLEV2>(d_comp, comp_bytes, d_blk_off, d_col_len, n_chunks, chunk_bytes, elem_bytes,
                                         d_out, out_bytes, d_chunk_status, ws, kNoAllocScratchBytes,
                                         reinterpret_cast<cudaStream_t>(stream));
}

extern "C" codag_status codag_set_tune(int codec, const codag_tune* tune) {
  if (codec < 0 || codec > 2 || !tune || !valid_warps(tune->warps_per_cta) || !valid_slots(tune->ring_slots) ||
      !valid_lut(tune->lut_bits))
    return CODAG_EINVAL;
  // an RLE v2 header with its data spans up to 2060 bytes; it must fit the window of
  // (slots - 1) KiB ahead of the read position
  if (codec != CODAG_CODEC_DEFLATE && tune->ring_slots < 4) return CODAG_EINVAL;
  if (tune->cta_per_chunk != 0 && tune->cta_per_chunk != 1) return CODAG_EINVAL;
  if (tune->table_global != 0) return CODAG_EINVAL;  // per-file calls: tables in shared memory (no workspace)
  // refused since a Deflate chunk per CTA meant pairs of warps
  if (codec == CODAG_CODEC_DEFLATE && tune->cta_per_chunk && (tune->warps_per_cta & 1)) return CODAG_EINVAL;
  std::lock_guard<std::mutex> g(g_mu);
  g_tune[codec] = *tune;
  return CODAG_OK;
}

extern "C" codag_status codag_get_tune(int codec, codag_tune* tune) {
  if (codec < 0 || codec > 2 || !tune) return CODAG_EINVAL;
  *tune = tune_of(codec);
  return CODAG_OK;
}

extern "C" codag_status codag_set_wait_limit(uint64_t cycles) {
  if (cycles == 0) return CODAG_EINVAL;
  std::lock_guard<std::mutex> g(g_mu);
  g_wait_cycles = cycles;
  return CODAG_OK;
}

extern "C" codag_status codag_selftest_wait_timeout(int32_t* d_status, codag_stream_t stream) {
  if (!d_status) return CODAG_EINVAL;
  clear_stale_error();
  k_selftest_timeout<<<1, 32, 0, reinterpret_cast<cudaStream_t>(stream)>>>(d_status, wait_of());
  return finish_launch();
}

