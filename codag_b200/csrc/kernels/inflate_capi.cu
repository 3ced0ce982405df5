// Deflate: the per-file kernel and its entry point (include/codag.h).
#include "capi_common.cuh"
#include "decode_deflate.cuh"

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
  if (allow_smem(k_inflate, sizeof(InflateTeam)) != cudaSuccess) return CODAG_ECUDA;
  if (n_chunks > 0x7fffffffull) return CODAG_EINVAL;
  k_inflate<<<static_cast<unsigned>(n_chunks), 32 * kTeamWarps, sizeof(InflateTeam), reinterpret_cast<cudaStream_t>(stream)>>>(
      d_comp, comp_bytes, d_blk_off, chunk_bytes, static_cast<uint32_t>(wrapper_bytes), d_out, out_bytes,
      d_chunk_status, wait_of());
  return finish_launch();
}
