// One-block-per-plane kernel of the real-plane solve (cvb_rp.cuh).  Built once per tensor type with
// -DCVB_IO=float | __nv_bfloat16 -DCVB_IO_NAME=f32 | bf16.
#include "../../include/converse_b200.h"
#include "cvb_internal.h"
#include "cvb_rp.cuh"

#define CVB_CAT_(a, b) a##_##b
#define CVB_CAT(a, b) CVB_CAT_(a, b)

namespace cvb {
namespace rp {

template <typename IO>
__global__ void __launch_bounds__(256, 3) plane_small_kernel(const __grid_constant__ Params P) {
  extern __shared__ float2 smem[];
  pdl_start();
  plane_body<IO, kSmallRadix>(P, smem);
}
template <typename IO>
__global__ void __launch_bounds__(512, 1) plane_kernel(const __grid_constant__ Params P) {
  extern __shared__ float2 smem[];
  pdl_start();
  plane_body<IO, kAnyRadix>(P, smem);
}

template <typename K>
static int go(K kernel, const Params& P, int threads, size_t smem, cudaStream_t st) {
  const int rc = allow_smem(kernel, smem);
  return rc != CVB_OK ? rc : launch_chained(kernel, dim3(P.nplane), threads, smem, st, P);
}
int CVB_CAT(launch_plane, CVB_IO_NAME)(const Params& P, bool small, int threads, size_t smem, cudaStream_t st) {
  return small ? go(plane_small_kernel<CVB_IO>, P, threads, smem, st) : go(plane_kernel<CVB_IO>, P, threads, smem, st);
}

}  // namespace rp
}  // namespace cvb
