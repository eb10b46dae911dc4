// Row kernel of the real-plane solve (cvb_rp.cuh), multi-launch form.
#include "../../include/converse_b200.h"
#include "cvb_internal.h"
#include "cvb_rp.cuh"

namespace cvb {
namespace rp {

__global__ void __launch_bounds__(256, 3) rows_small_kernel(const __grid_constant__ Params P) {
  extern __shared__ float2 smem[];
  pdl_start();
  rows_body<kSmallRadix, 0>(P, smem);
}
__global__ void __launch_bounds__(256, 2) rows_kernel(const __grid_constant__ Params P) {
  extern __shared__ float2 smem[];
  pdl_start();
  rows_body<kAnyRadix, 0>(P, smem);
}

template <typename K>
static int go(K kernel, const Params& P, int grid, int threads, size_t smem, cudaStream_t st) {
  const int rc = allow_smem(kernel, smem);
  return rc != CVB_OK ? rc : launch_chained(kernel, dim3(grid), threads, smem, st, P);
}
int launch_rows(const Params& P, bool small, int threads, int grid, size_t smem, cudaStream_t st) {
  if (small) return go(rows_small_kernel, P, grid, threads, smem, st);
  return go(rows_kernel, P, grid, threads, smem, st);
}

}  // namespace rp
}  // namespace cvb
