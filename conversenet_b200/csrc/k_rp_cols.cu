// Column kernels and upsampling epilogue of the real-plane solve (cvb_rp.cuh), multi-launch form.  Built once per
// tensor type with -DCVB_IO=float | __nv_bfloat16 -DCVB_IO_NAME=f32 | bf16.
#include "../../include/converse_b200.h"
#include "cvb_internal.h"
#include "cvb_rp.cuh"

#define CVB_CAT_(a, b) a##_##b
#define CVB_CAT(a, b) CVB_CAT_(a, b)

namespace cvb {
namespace rp {

// Small radices: 24 warps on an SM (80 registers); any radix: 128 registers.
template <typename IO>
__global__ void __launch_bounds__(256, 3) cols_fwd_small_kernel(const __grid_constant__ Params P) {
  extern __shared__ float2 smem[];
  pdl_start();
  cols_fwd_body<IO, kSmallRadix, 0>(P, smem);
}
template <typename IO>
__global__ void __launch_bounds__(256, 3) cols_inv_small_kernel(const __grid_constant__ Params P) {
  extern __shared__ float2 smem[];
  pdl_start();
  cols_inv_body<IO, kSmallRadix, 0>(P, smem);
}
template <typename IO>
__global__ void __launch_bounds__(256, 2) cols_fwd_kernel(const __grid_constant__ Params P) {
  extern __shared__ float2 smem[];
  pdl_start();
  cols_fwd_body<IO, kAnyRadix, 0>(P, smem);
}
template <typename IO>
__global__ void __launch_bounds__(256, 2) cols_inv_kernel(const __grid_constant__ Params P) {
  extern __shared__ float2 smem[];
  pdl_start();
  cols_inv_body<IO, kAnyRadix, 0>(P, smem);
}
template <typename IO>
__global__ void __launch_bounds__(128) epilogue_kernel(const __grid_constant__ Params P) {
  __shared__ __align__(16) unsigned char band[kEpiBand];
  pdl_start();
  epilogue_body<IO>(P, band);
}

template <typename K>
static int go(K kernel, const Params& P, int grid, int threads, size_t smem, cudaStream_t st) {
  const int rc = allow_smem(kernel, smem);
  return rc != CVB_OK ? rc : launch_chained(kernel, dim3(grid), threads, smem, st, P);
}
int CVB_CAT(launch_cols_fwd, CVB_IO_NAME)(const Params& P, bool small, int threads, int grid, size_t smem, cudaStream_t st) {
  if (small) return go(cols_fwd_small_kernel<CVB_IO>, P, grid, threads, smem, st);
  return go(cols_fwd_kernel<CVB_IO>, P, grid, threads, smem, st);
}
int CVB_CAT(launch_cols_inv, CVB_IO_NAME)(const Params& P, bool small, int threads, int grid, size_t smem, cudaStream_t st) {
  if (small) return go(cols_inv_small_kernel<CVB_IO>, P, grid, threads, smem, st);
  return go(cols_inv_kernel<CVB_IO>, P, grid, threads, smem, st);
}
int CVB_CAT(launch_epilogue, CVB_IO_NAME)(const Params& P, cudaStream_t st) {
  return launch_chained(epilogue_kernel<CVB_IO>, dim3((P.H + kEpiRows - 1) / kEpiRows, P.nplane), 128, 0, st, P);
}

}  // namespace rp
}  // namespace cvb
