// The final sum's kernel and entry point (msm_final.cuh has the method and the device code).
#include "msm_final.cuh"
#include "pointer_access.h"

#include <cooperative_groups.h>
#include <cuda_runtime.h>

namespace msm_b200 {

__global__ void __cluster_dims__(FINAL_BLOCKS, 1, 1) __launch_bounds__(FINAL_THREADS)
    final_sum_kernel(const jacobian *__restrict__ results, msm_b200_affine_point *point) {
  __shared__ final_shared sh;
  final_sum_block(sh, cooperative_groups::this_cluster(), results, point);
}

// A pointer the kernel can dereference (pointer_access.h): device memory of
// the current device or of a peer it has access to, managed memory, or pinned
// host memory through its device alias; anything else is refused.
static cudaError_t device_view(const void *ptr, void **view) {
  int device = 0;
  cudaError_t err = cudaGetDevice(&device);
  if (err != cudaSuccess)
    return err;
  cudaPointerAttributes attr{};
  if ((err = cudaPointerGetAttributes(&attr, ptr)) != cudaSuccess)
    return err;
  const bool peer = attr.type == cudaMemoryTypeDevice && attr.device != device && peer_access_recorded(device, attr.device);
  return kernel_view(ptr, attr, device, peer, host_memory::device_alias, view);
}

cudaError_t final_sum(const void *results, msm_b200_affine_point *point, cudaStream_t stream) {
  if (!results || !point || reinterpret_cast<uintptr_t>(results) % 16 || reinterpret_cast<uintptr_t>(point) % 4)
    return cudaErrorInvalidValue;
  void *r = nullptr, *p = nullptr;
  cudaError_t err = device_view(results, &r);
  if (err == cudaSuccess)
    err = device_view(point, &p);
  if (err != cudaSuccess)
    return err;
  final_sum_kernel<<<FINAL_BLOCKS, FINAL_THREADS, 0, stream>>>(static_cast<const jacobian *>(r), static_cast<msm_b200_affine_point *>(p));
  return cudaGetLastError();
}

} // namespace msm_b200

extern "C" bc_error msm_b200_final_sum_async(const void *results, msm_b200_affine_point *point, bc_stream stream) {
  return static_cast<bc_error>(msm_b200::final_sum(results, point, static_cast<cudaStream_t>(stream.handle)));
}
