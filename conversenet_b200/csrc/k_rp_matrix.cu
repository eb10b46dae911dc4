// Strip kernels of the real-plane solve whose R0-point transform is a matrix stage (lengths with a large prime).  Built
// once per width with -DCVB_MP=..; 128 threads, as many blocks on an SM as the pairs held in registers allow.
#include "../../include/converse_b200.h"
#include "cvb_internal.h"
#include "cvb_rp_bwd.cuh"

#define CVB_CAT_(a, b) a##_##b
#define CVB_CAT(a, b) CVB_CAT_(a, b)
// 256 threads where registers allow two such blocks, else 128 and three blocks
#define CVB_RP_THREADS (CVB_MP <= 44 ? 256 : 128)
#define CVB_RP_BLOCKS (CVB_MP <= 44 ? 2 : 3)

namespace cvb {
namespace rp {

template <typename IO, int MP>
__global__ void __launch_bounds__(CVB_RP_THREADS, CVB_RP_BLOCKS) matrix_cols_fwd_kernel(const __grid_constant__ Params P) {
  extern __shared__ float2 smem[];
  pdl_start();
  cols_fwd_body<IO, kMatrixR1, MP>(P, smem);
}
template <int MP>
__global__ void __launch_bounds__(CVB_RP_THREADS, CVB_RP_BLOCKS) matrix_rows_kernel(const __grid_constant__ Params P) {
  extern __shared__ float2 smem[];
  pdl_start();
  rows_body<kMatrixR1, MP>(P, smem);
}
template <typename IO, int MP>
__global__ void __launch_bounds__(CVB_RP_THREADS, CVB_RP_BLOCKS) matrix_cols_inv_kernel(const __grid_constant__ Params P) {
  extern __shared__ float2 smem[];
  pdl_start();
  cols_inv_body<IO, kMatrixR1, MP>(P, smem);
}

template <int MP>
__global__ void __launch_bounds__(128, 3) matrix_rows_bwd_kernel(const __grid_constant__ BwdParams Q) {
  extern __shared__ float2 smem[];
  pdl_start();
  rows_bwd_body<kMatrixR1, MP>(Q, smem);
}

template <typename K>
static int go(K kernel, const Params& P, int threads, int grid, size_t smem, cudaStream_t st) {
  const int rc = allow_smem(kernel, smem);
  return rc != CVB_OK ? rc : launch_chained(kernel, dim3(grid), threads < CVB_RP_THREADS ? threads : CVB_RP_THREADS, smem, st, P);
}
int CVB_CAT(launch_matrix_cols_fwd, CVB_MP)(const Params& P, int io_dtype, int threads, int grid, size_t smem, cudaStream_t st) {
  return io_dtype == CVB_F32 ? go(matrix_cols_fwd_kernel<float, CVB_MP>, P, threads, grid, smem, st)
                             : go(matrix_cols_fwd_kernel<__nv_bfloat16, CVB_MP>, P, threads, grid, smem, st);
}
int CVB_CAT(launch_matrix_rows, CVB_MP)(const Params& P, int, int threads, int grid, size_t smem, cudaStream_t st) {
  return go(matrix_rows_kernel<CVB_MP>, P, threads, grid, smem, st);
}
int CVB_CAT(launch_matrix_cols_inv, CVB_MP)(const Params& P, int io_dtype, int threads, int grid, size_t smem, cudaStream_t st) {
  return io_dtype == CVB_F32 ? go(matrix_cols_inv_kernel<float, CVB_MP>, P, threads, grid, smem, st)
                             : go(matrix_cols_inv_kernel<__nv_bfloat16, CVB_MP>, P, threads, grid, smem, st);
}

int CVB_CAT(launch_matrix_rows_bwd, CVB_MP)(const BwdParams& Q, dim3 grid, size_t smem, cudaStream_t st) {
  if (const int rc = allow_smem(matrix_rows_bwd_kernel<CVB_MP>, smem)) return rc;
  matrix_rows_bwd_kernel<CVB_MP><<<grid, 128, smem, st>>>(Q);
  CVB_CUDA(cudaGetLastError());
  return CVB_OK;
}

}  // namespace rp
}  // namespace cvb
