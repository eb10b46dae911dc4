// Internal glue between the translation units of libconverse_b200.so.
#pragma once
#include "cvb_kernels.cuh"
#include "cvb_plan.h"

namespace cvb {

// Records a failing CUDA runtime call for cvb_last_cuda_error and returns CVB_ERR_CUDA.
int cuda_fail(cudaError_t e);

#define CVB_CUDA(call)                                   \
  do {                                                   \
    cudaError_t e__ = (call);                            \
    if (e__ != cudaSuccess) return ::cvb::cuda_fail(e__); \
  } while (0)

#ifdef __CUDACC__
// Launch with programmatic dependent launch: the kernel (it calls pdl_start() first) may be placed on SMs that the kernel
// before it has left, which hides the launch gap of back-to-back kernels (16 x 64 planes of 68 x 68 upsampled by 2, call after
// call: 38.9 -> 37.6 us with the pair table, 40.7 -> 38.9 us with the real-plane one).
template <typename... P, typename... A>
int launch_chained(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, const A&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = dim3(threads); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at; cfg.numAttrs = 1;
  CVB_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
  return CVB_OK;
}
// Dynamic shared memory beyond 48 KB has to be allowed.  The limit belongs to the kernel and not to the launch: it is always
// all there is (none of these kernels has static shared memory), since a smaller call's size, set by another thread between
// this one and the launch, would make the launch fail.
template <typename... P>
int allow_smem(void (*kernel)(P...), size_t smem) {
  if (smem <= 48 * 1024) return CVB_OK;
  CVB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit));
  return CVB_OK;
}
#endif

// Tuning aids read the environment only in tuning builds (-DCVB_TUNING); a shipped library ignores them.
#ifdef CVB_TUNING
int env_int(const char* name, int dflt);
#define CVB_TUNE(name, dflt) ::cvb::env_int(name, dflt)
#else
#define CVB_TUNE(name, dflt) (dflt)
#endif

// Process-wide routing options (cvb_set_option / cvb_get_option in the C ABI).
int option(int which);
int sm_count();  // multiprocessors of the current device
int* status_ptr();  // the current device's status word (null: cannot be had)

// Number of (channel, batch-pair) work items = blocks of the shared-memory kernels.
inline int num_pairs(const FwdParams& P) { return P.C * ((P.B + 1) / 2); }

// Runtime-plan kernel (k_dynamic.cu).
int launch_dynamic(const FwdParams& P, int io_dtype, size_t smem, cudaStream_t st);
int launch_xspec(const XspecParams& Q, cudaStream_t st);
int launch_tap_gradient(const float* g, const float* r, float* out, int nseg, int B, int C, int h, int w, int k,
                        int s, cudaStream_t st);

// Multi-pass path through a workspace (k_strip.cu).
int launch_strip(const FwdParams& P, int io_dtype, void* workspace, size_t ws_bytes, cudaStream_t st);
// Same kernels, workspace = the library's own fixed device array (no allocation anywhere).
int static_scratch_address(void** out);
int launch_strip_static_scratch(const FwdParams& P, int io_dtype, cudaStream_t st);

// Real-plane solve for every size with a two-stage plan (k_rp.cu).
namespace rp {
struct Params;
struct Route;
size_t table_bytes(int C, int h, int w);
int build_table(const float* weight, const float* bias, int C, int k, int s, int h, int w, float eps, int kind,
                void* table, cudaStream_t st);
int cols_fwd(Params& P, int planes, cudaStream_t st);
int rows(Params& P, int planes, cudaStream_t st);
int cols_inv(Params& P, int planes, cudaStream_t st);
size_t bwd_workspace(int B, int C, int H, int W, int k, int s, int p, bool want_x, bool want_params, int sms);
int run_bwd(const float* x, const float* g, const float* r, const void* table, const float* weight, const float* bias,
            float* gx, float* gw, float* gb, int B, int C, int H, int W, int k, int s, int p, int pad_mode, float eps,
            void* workspace, size_t ws_bytes, int sms, cudaStream_t st);
int run(Params& P, const Route& r, int io_dtype, void* workspace, size_t ws_bytes, cudaStream_t st);
}  // namespace rp

// Fused channel-mixing kernels of ConverseBlock (k_block.cu).
struct BlockParams;
int launch_ln_pw_gelu(const BlockParams& P, int io_dtype, cudaStream_t st);
int launch_pw_res_mlp(const BlockParams& P, int io_dtype, int sms, cudaStream_t st);
// tcgen05 variant of the first kernel (k_block_tc.cu): fp32, HW a multiple of 128
int launch_ln_pw_gelu_tc(const BlockParams& P, int sms, int* status, cudaStream_t st);
// tcgen05: out = res + alpha * (W . t + b), 128 -> 64 channels (P.t, P.x = res, P.w_a, P.b_a, P.alpha1)
int launch_pw_res_tc(const BlockParams& P, int sms, int* status, cudaStream_t st);
// warp-specialised, double-buffered versions of the two (k_block_tc2.cu)
int launch_ln_pw_gelu_tc2(const BlockParams& P, int io_dtype, int sms, int* status, cudaStream_t st);
int launch_pw_res_tc2(const BlockParams& P, int io_dtype, int sms, int* status, cudaStream_t st);
int launch_ln_pw_gelu_tc3(const BlockParams& P, int io_dtype, int sms, int* status, cudaStream_t st);
int launch_pw_res_tc3(const BlockParams& P, int io_dtype, int sms, int* status, cudaStream_t st);

// packed weights, both sides of the block (k_block_mlp.cu)
size_t block_pack_bytes();
int launch_block_pack(const float* ln1_w, const float* ln1_b, const float* w1, const float* b1, const float* w2,
                      const float* b2, const float* a1, const float* ln2_w, const float* ln2_b, const float* w3,
                      const float* b3, const float* w4, const float* b4, const float* a2, void* pack, cudaStream_t st);
int launch_block_mix(bool post, const void* x, const void* t, void* out, const void* pack, float eps, int B, int HW,
                     int io_dtype, int sms, int* status, cudaStream_t st);

int launch_block_mix_train(bool post, const float* x, const float* t, float* out, float* z, float* x1, const void* pack,
                           float eps, int B, int HW, int sms, int* status, cudaStream_t st);
// gradients of the block (k_block_train.cu); `conv`: the gradient of its Converse2D
size_t block_grad_floats();
size_t block_grad_workspace(int B, int HW, size_t conv_ws, int sms);
int run_block_grad(const cvb_block_bwd_args& A, size_t conv_ws, int sms, int* status, cudaStream_t st,
                   int (*conv)(const cvb_block_bwd_args&, const float* gu, float* gt, void* ws, size_t bytes));

// Multi-pass kernels with a compile-time axis plan (k_strip2.cu, one object per registry line).
struct StripParams;
typedef int (*Strip2Launcher)(const StripParams& SP, int io_dtype, cudaStream_t st);
typedef int (*Strip2Resident)(int io_dtype, int k, int* blocks_per_sm);  // [3]: kernels A, B, C
struct Strip2Entry {
  int r0, r1, s0, s1;  // axis length r0 * r1; Rader sub-plan s0 * s1 of r0 - 1 (0, 0 if r0 is a register radix)
  Strip2Launcher A, B, C;
  Strip2Resident Q;
};

// Tensor-core multi-pass kernels (k_gemmdft.cu, one object per registry line).
namespace gd { struct Params; }
typedef int (*GdLauncher)(const gd::Params& P, int io_dtype, cudaStream_t st);
struct GdEntry {
  int r0;
  GdLauncher A, B1, B2, C;
};

// Compile-time-plan kernels (k_static.cu, one object per registry line).
typedef int (*StaticLauncher)(const FwdParams& P, int io_dtype, size_t smem, int blocks, cudaStream_t st);
struct StaticEntry {
  int ry0, ry1, rx0, rx1, nt, mb;
  StaticLauncher fn;          // one block per plane pair
  StaticLauncher fn_persist;  // persistent blocks with prefetch
};

}  // namespace cvb
