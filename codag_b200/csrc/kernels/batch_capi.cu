// Batched persistent decompression (include/codag.h, codag_batch_*): one launch over many
// independent streams of uneven size and mixed codec.
#include <algorithm>
#include <cstdint>
#include <mutex>
#include <new>
#include <utility>
#include <vector>

#include "capi_common.cuh"
#include "decode_deflate.cuh"
#include "decode_rle.cuh"

using namespace codag_dev;
using namespace codag_capi;

namespace {

constexpr uint32_t kWarps = 8;       // warps per CTA: a Deflate team uses six, the RLE files all
constexpr uint32_t kRleFirst = 3;    // with both kinds of work, every 3rd CTA takes RLE files first
using RleRing = InRing<4>;
struct BatchShared {
  union {
    InflateTeam team;
    alignas(128) uint8_t ring[kWarps][RleRing::kBytes];  // overlays the team's window only
  };
  uint64_t bar[kWarps][4];  // the RLE rings' barriers (the team has its own)
};
static_assert(kWarps * RleRing::kBytes <= sizeof(InflateTeam::win), "the team's barriers keep their place");
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

// An RLE stream on one warp.  Values go straight to global memory: element by element when the
// output is element aligned, byte by byte otherwise.
__device__ __forceinline__ int rle_job(const BatchArgs& a, const codag_chunk_desc& d, RleRing& in, uint32_t lane) {
  if (!job_in_bounds(a, d)) return CODAG_ECORRUPT;
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

__device__ __forceinline__ void rle_ring(RleRing& in, BatchShared& sh, uint64_t wait_cycles, uint32_t warp,
                                         uint32_t lane) {
  in.buf = sh.ring[warp];
  in.sbuf = smem_u32(in.buf);
  in.bar = sh.bar[warp];
  in.phase = 0;
  in.wait_cycles = wait_cycles;
  in.lane = lane;
  init_ring_barriers<4>(in.bar, lane);
}

// Entries [0, n) of the order, taken by the CTA's first six warps together: a Deflate stream by the
// team, anything else by its first warp alone (in the window's memory, which is idle then).
__device__ __forceinline__ void team_jobs(const BatchArgs& a, uint64_t n, uint32_t* queue, BatchShared& sh,
                                          uint64_t wait_cycles, uint32_t warp, uint32_t lane, RleRing& rle) {
  InflateTeam& sm = sh.team;
  InflateRing in;
  TokenRing tin;
  InflateWin o;
  inflate_rings(in, tin, sm, wait_cycles, warp, lane);
  inflate_window(o, sm, lane);
  for (;;) {
    if (warp == 0 && lane == 0) {
      sm.job = atomicAdd(queue, 1u);
      sm.stop = sm.dead = 0;
      sm.status = CODAG_OK;
    }
    job_barrier();
    const uint32_t k = sm.job;
    if (k >= n) break;
    const uint32_t i = a.order ? a.order[k] : k;
    const codag_chunk_desc d = a.descs[i];
    if (d.codec != CODAG_CODEC_DEFLATE) {
      if (warp == 0) {
        const int st = rle_job(a, d, rle, lane);
        if (lane == 0) {
          if (a.status) a.status[i] = st;
          sm.status = st;
        }
        fence_proxy_async_smem();
      }
    } else if (!job_in_bounds(a, d)) {
      if (a.status && warp == 0 && lane == 0) a.status[i] = CODAG_ECORRUPT;
    } else {
      if (warp < 2) {
        in.begin(a.comp + d.comp_off, d.comp_len);
        inflate_scan(in, sm, d.wrapper_bytes, warp, lane);
      } else if (warp < 4) {
        tin.begin(a.comp + d.comp_off, d.comp_len);
        inflate_tokens(tin, sm, warp - 2u, lane);
      } else if (warp == 4) {
        inflate_place(sm, d.out_len, lane);
      } else {
        o.begin(a.out + d.out_off, d.out_len);
        const int st = inflate_copy(sm, o, lane);
        if (a.status && lane == 0) a.status[i] = st;
      }
    }
    job_barrier();
    const bool timed_out = sm.status == CODAG_ETIMEOUT || sm.dead;
    job_barrier();  // every warp has looked before the next job resets it
    if (timed_out) break;  // ring state unknown: the team stops
  }
}

// RLE entries [n0, n) of the order, one per warp.
__device__ __forceinline__ void rle_jobs(const BatchArgs& a, uint64_t n0, uint64_t n, uint32_t* queue, uint32_t lane,
                                         RleRing& in) {
  for (;;) {
    uint32_t k = 0;
    if (lane == 0) k = atomicAdd(queue, 1u);
    k = __shfl_sync(FULL, k, 0);
    if (k >= n - n0) break;
    const uint32_t i = a.order[n0 + k];
    const int st = rle_job(a, a.descs[i], in, lane);
    if (a.status && lane == 0) a.status[i] = st;
    if (st == CODAG_ETIMEOUT) break;  // ring state unknown: this warp stops pulling work
  }
}

// Persistent grid, three CTAs per SM.  The first n_team entries of the order are taken by teams
// (queue[0]), the others, RLE files of a plan, by single warps (queue[1]).  A CTA does both: most start
// with the team's entries and turn all eight warps to RLE files when those run out; every
// kRleFirst-th begins with the RLE files, so that the longest of both kinds start at once.
__global__ void __launch_bounds__(32 * kWarps, 3)
    k_batch(BatchArgs a, uint64_t n, uint64_t n_team, uint32_t* __restrict__ queue, uint64_t wait_cycles) {
  extern __shared__ __align__(128) uint8_t smem[];
  BatchShared& sh = *reinterpret_cast<BatchShared*>(smem);
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  RleRing rle;
  rle_ring(rle, sh, wait_cycles, warp, lane);
  const bool rle_first = blockIdx.x % kRleFirst == kRleFirst - 1u;
  for (uint32_t phase = 0; phase < 2; phase++) {
    if ((phase == 0) == rle_first) {
      if (n_team < n) rle_jobs(a, n_team, n, queue + 1, lane, rle);
    } else if (n_team && warp < kTeamWarps) {
      team_jobs(a, n_team, queue, sh, wait_cycles, warp, lane, rle);
    }
    __syncthreads();  // the phases share the memory
    fence_proxy_async_smem();
  }
}

}  // namespace

struct codag_plan {
  uint64_t n = 0;
  uint64_t n_team = 0;  // leading entries of the order taken by teams: the Deflate files
  codag_chunk_desc* d_descs = nullptr;
  uint32_t* d_order = nullptr;
  uint32_t* d_queue = nullptr;
  int grid = 0;
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
  if (allow_smem(k_batch, sizeof(BatchShared)) != cudaSuccess) return CODAG_ECUDA;
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return CODAG_ECUDA;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch, 32 * kWarps, sizeof(BatchShared)) != cudaSuccess)
    return CODAG_ECUDA;
  *cap = sms * std::max(per_sm, 1);
  return CODAG_OK;
}

void batch_enqueue(const BatchArgs& a, uint64_t n, uint64_t n_team, uint32_t* queue, int grid, cudaStream_t s) {
  cudaMemsetAsync(queue, 0, (n_team < n ? 2 : 1) * sizeof(uint32_t), s);
  k_batch<<<grid, 32 * kWarps, sizeof(BatchShared), s>>>(a, n, n_team, queue, wait_of());
}

// Work estimate that orders the queue within a kind of work: compressed bytes, and for RLE files,
// whose runs expand at store speed, a share of the output.
uint64_t chunk_cost(const codag_chunk_desc& d) {
  return d.codec == CODAG_CODEC_DEFLATE ? 8ull * d.comp_len + d.out_len : static_cast<uint64_t>(d.comp_len) + d.out_len / 4;
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
  auto team = [&](uint32_t i) { return h_descs[i].codec == CODAG_CODEC_DEFLATE; };
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
  int cap = 0;
  const codag_status st = batch_grid_cap(&cap);
  if (st != CODAG_OK) {
    codag_batch_destroy(p);
    return st;
  }
  const uint64_t need = p->n_team + (n - p->n_team + kWarps - 1) / kWarps;
  p->grid = static_cast<int>(std::min<uint64_t>(need, static_cast<uint64_t>(cap)));
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
    batch_enqueue(args, p->n, p->n_team, p->d_queue, p->grid, s);
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
      batch_enqueue(args, p->n, p->n_team, p->d_queue, p->grid, cap);
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

// The host does not know the codecs here, so teams take every entry.
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
  batch_enqueue(args, n, n, d_queue, static_cast<int>(std::min<uint64_t>(n, static_cast<uint64_t>(cap))),
                reinterpret_cast<cudaStream_t>(stream));
  return finish_launch();
}
