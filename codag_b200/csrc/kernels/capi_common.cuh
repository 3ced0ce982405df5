// Shared by the translation units of libcodag_b200.so: chunk geometry on the device, and on the
// host the launch helpers and the process-wide settings (defined in codag_capi.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>

#include "device_common.cuh"

namespace codag_dev {

__device__ __forceinline__ uint64_t store_bytes(uint64_t base, uint64_t chunk_bytes, uint64_t out_bytes) {
  return base < out_bytes ? (chunk_bytes < out_bytes - base ? chunk_bytes : out_bytes - base) : 0;
}

__device__ __forceinline__ bool valid_elem_dev(uint32_t e) { return e == 1 || e == 2 || e == 4 || e == 8; }

__device__ __forceinline__ bool stream_in_bounds(uint64_t off, uint64_t len, uint64_t comp_bytes) {
  return off <= comp_bytes && len <= comp_bytes - off && len < (1ull << 28);
}

}  // namespace codag_dev

namespace codag_capi {

inline bool valid_slots(int s) { return s == 2 || s == 4 || s == 8; }
inline bool valid_lut(int b) { return b == 9 || b == 10 || b == 11; }
inline bool valid_warps(int w) { return w >= 1 && w <= 8; }
inline bool valid_elem(int e) { return e == 1 || e == 2 || e == 4 || e == 8; }

uint64_t wait_of();  // bound of a device wait, in clock cycles (codag_set_wait_limit)

// Raises a kernel's dynamic shared-memory limit to at least `bytes` on the current device.  The
// limit is per kernel and one instantiation serves shapes of different sizes, so it is only
// ever raised: lowering it for a small shape would make a later launch of a larger one, or a
// plan made earlier, fail.
cudaError_t allow_smem_of(const void* kernel, uint32_t bytes);
template <class K>
cudaError_t allow_smem(K kernel, uint32_t bytes) {
  return allow_smem_of(reinterpret_cast<const void*>(kernel), bytes);
}

// An entry point clears a CUDA error that earlier work of the process left pending (for
// example an allocation that a caching allocator retried after freeing memory), so that the
// check after its own launches reports only errors of those launches.
inline void clear_stale_error() { (void)cudaGetLastError(); }

inline codag_status finish_launch() {
  const cudaError_t err = cudaGetLastError();
  if (err == cudaSuccess) return CODAG_OK;
  std::fprintf(stderr, "codag: kernel launch failed: %s\n", cudaGetErrorName(err));
  return CODAG_ECUDA;
}

}  // namespace codag_capi
