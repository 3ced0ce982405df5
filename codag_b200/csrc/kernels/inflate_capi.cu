// Deflate: the per-file kernel and its entry point (include/codag.h).
#include "capi_common.cuh"
#include "decode_deflate_warp.cuh"

using namespace codag_dev;
using namespace codag_capi;

namespace {

// One team per chunk and CTA.
__global__ void __launch_bounds__(32 * kTeamWarps, 3)
    k_inflate(const uint8_t* __restrict__ comp, uint64_t comp_bytes, const uint64_t* __restrict__ blk_off,
              uint64_t chunk_bytes, uint32_t wrapper, uint8_t* __restrict__ out, uint64_t out_bytes,
              int32_t* __restrict__ status, uint64_t wait_cycles) {
  extern __shared__ __align__(128) uint8_t smem[];
  InflateTeam& sm = *reinterpret_cast<InflateTeam*>(smem);
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint64_t chunk = blockIdx.x;
  const uint64_t off = blk_off[chunk], next = blk_off[chunk + 1];
  if (next < off || !stream_in_bounds(off, next - off, comp_bytes)) {
    if (status && threadIdx.x == 0) status[chunk] = CODAG_ECORRUPT;
    return;
  }
  if (threadIdx.x == 0) sm.stop = sm.dead = 0;
  __syncthreads();
  InflateRing in;
  TokenRing tin;
  inflate_rings(in, tin, sm, wait_cycles, warp, lane);
  if (warp < 2) {
    in.begin(comp + off, static_cast<uint32_t>(next - off));
    inflate_scan(in, sm, wrapper, warp, lane);
  } else if (warp < 4) {
    tin.begin(comp + off, static_cast<uint32_t>(next - off));
    inflate_tokens(tin, sm, warp - 2u, lane);
  } else if (warp == 4) {
    inflate_place(sm, chunk_bytes, lane);
  } else {
    const uint64_t base = chunk * chunk_bytes;
    InflateWin o;
    inflate_window(o, sm, lane);
    o.begin(out + base, store_bytes(base, chunk_bytes, out_bytes));
    const int st = inflate_copy(sm, o, comp + off, static_cast<uint32_t>(next - off), lane);
    if (status && lane == 0) status[chunk] = st;
  }
}

// One warp per chunk, kWarpsPerCta in a CTA.
constexpr uint32_t kWarpsPerCta = 2;
struct WarpShared {
  alignas(128) uint8_t ring[align16(InRing<2>::kAlloc)];
  alignas(16) uint8_t win[InflateWarpWin::kBytes];
  InflateWarp tables;
  uint64_t bar[2];
};
__global__ void __launch_bounds__(32 * kWarpsPerCta, 16)
    k_inflate_warp(const uint8_t* __restrict__ comp, uint64_t comp_bytes, const uint64_t* __restrict__ blk_off, uint64_t n_chunks,
                   uint64_t chunk_bytes, uint32_t wrapper, uint8_t* __restrict__ out, uint64_t out_bytes,
                   int32_t* __restrict__ status, uint64_t wait_cycles) {
  __shared__ WarpShared shared[kWarpsPerCta];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint64_t chunk = static_cast<uint64_t>(blockIdx.x) * kWarpsPerCta + warp;
  if (chunk >= n_chunks) return;
  WarpShared& sh = shared[warp];
  const uint64_t off = blk_off[chunk], next = blk_off[chunk + 1];
  int st = CODAG_ECORRUPT;
  if (next >= off && stream_in_bounds(off, next - off, comp_bytes)) {
    InRing<2> in;
    bind_ring(in, sh.ring, sh.bar, wait_cycles, lane, true);
    in.begin(comp + off, static_cast<uint32_t>(next - off));
    InflateWarpWin o;
    o.buf = sh.win;
    o.sbuf = smem_u32(sh.win);
    o.lane = lane;
    const uint64_t base = chunk * chunk_bytes;
    o.begin(out + base, store_bytes(base, chunk_bytes, out_bytes));
    st = inflate_warp(in, o, sh.tables, chunk_bytes, wrapper, lane);
  }
  if (status && lane == 0) status[chunk] = st;
}

codag_status launch_warp(const uint8_t* comp, uint64_t comp_bytes, const uint64_t* blk_off, uint64_t n, uint64_t chunk_bytes,
                         uint32_t wrapper, uint8_t* out, uint64_t out_bytes, int32_t* status, cudaStream_t s) {
  const uint64_t grid = (n + kWarpsPerCta - 1) / kWarpsPerCta;
  if (grid > 0x7fffffffull) return CODAG_EINVAL;
  k_inflate_warp<<<static_cast<unsigned>(grid), 32 * kWarpsPerCta, 0, s>>>(comp, comp_bytes, blk_off, n, chunk_bytes, wrapper,
                                                                                 out, out_bytes, status, wait_of());
  return finish_launch();
}

// Whether a warp each is faster than a team each for n chunks, by the mean length of their streams (from comp_bytes: too
// long for a part of a file, and then no reason for warps).  Measured, us, team | warp, text: 200 chunks of 1 KiB
// 57 | 152, 4096 415 | 220, 1024 of 4 KiB 175 | 480, 16384 2063 | 2433; zeros: 1024 of 4 KiB 122 | 42, of 64 KiB
// 329 | 210, 512 of 128 KiB 283 | 370; random bytes: 1024 of 4 KiB 31 | 23, 512 of 128 KiB 155 | 263.
bool warp_pays(uint64_t n, uint64_t chunk_bytes, uint64_t comp_bytes) {
  constexpr float kSms = 148;
  const InflateCost c = inflate_cost(chunk_bytes, comp_bytes / n);
  const float count = static_cast<float>(n), teams = count / (3 * kSms), warps = 1.6f * count / (32 * kSms);
  return c.warp * (warps > 1 ? warps : 1) < 4000.f + c.team * (teams > 1 ? teams : 1);
}

}  // namespace

extern "C" codag_status codag_decompress_deflate(const uint8_t* d_comp, uint64_t comp_bytes, const uint64_t* d_blk_off,
                                                 uint64_t n_chunks, uint64_t chunk_bytes, int wrapper_bytes,
                                                 uint8_t* d_out, uint64_t out_bytes, int32_t* d_chunk_status,
                                                 codag_stream_t stream) {
  if (!d_comp || !d_blk_off || (!d_out && out_bytes) || chunk_bytes == 0 || chunk_bytes >= (1ull << 31) ||
      wrapper_bytes < 0 || wrapper_bytes > 16)
    return CODAG_EINVAL;
  if (n_chunks == 0) return CODAG_OK;
  clear_stale_error();
  if (warp_pays(n_chunks, chunk_bytes, comp_bytes)) {
    return launch_warp(d_comp, comp_bytes, d_blk_off, n_chunks, chunk_bytes, static_cast<uint32_t>(wrapper_bytes), d_out, out_bytes,
                  d_chunk_status, reinterpret_cast<cudaStream_t>(stream));
  }
  if (allow_smem(k_inflate, sizeof(InflateTeam)) != cudaSuccess) return CODAG_ECUDA;
  if (n_chunks > 0x7fffffffull) return CODAG_EINVAL;
  k_inflate<<<static_cast<unsigned>(n_chunks), 32 * kTeamWarps, sizeof(InflateTeam), reinterpret_cast<cudaStream_t>(stream)>>>(
      d_comp, comp_bytes, d_blk_off, chunk_bytes, static_cast<uint32_t>(wrapper_bytes), d_out, out_bytes,
      d_chunk_status, wait_of());
  return finish_launch();
}
