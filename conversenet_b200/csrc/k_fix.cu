// Strip kernels of the real-plane solve as integer contractions on the tensor cores (cvb_fix.cuh).
#include "../../include/converse_b200.h"
#include "cvb_internal.h"
#include "cvb_rp_plan.h"

namespace cvb {
namespace rp {

template <int KIND, typename IO, bool EXTRA>
__global__ void __launch_bounds__(kFixThreads, 1) fix_kernel(const __grid_constant__ Params P) {
  extern __shared__ __align__(128) unsigned char fix_smem_raw[];
  pdl_start();
  fix_body<KIND, IO, EXTRA>(P, fix_smem_raw);
}

template <int KIND, typename IO>
static int go(const Params& P, int sms, cudaStream_t st) {
  const int n = KIND == kFixRows ? P.ax.n : P.ay.n;
  const int tiles = (fix_lines(KIND, P) + kFixLines - 1) / kFixLines;
  auto kernel = n >= 256 ? fix_kernel<KIND, IO, true> : fix_kernel<KIND, IO, false>;
  const size_t smem = fix_smem(KIND, n);
  const int rc = allow_smem(kernel, smem);
  return rc != CVB_OK ? rc : launch_chained(kernel, dim3(tiles < sms ? tiles : sms), kFixThreads, smem, st, P);
}
int launch_fix(int kind, const Params& P, int io_dtype, int sms, cudaStream_t st) {
  const bool f32 = io_dtype == CVB_F32;
  if (kind == kFixRows) return go<kFixRows, float>(P, sms, st);
  if (kind == kFixFwd) return f32 ? go<kFixFwd, float>(P, sms, st) : go<kFixFwd, __nv_bfloat16>(P, sms, st);
  return f32 ? go<kFixInv, float>(P, sms, st) : go<kFixInv, __nv_bfloat16>(P, sms, st);
}

}  // namespace rp
}  // namespace cvb
