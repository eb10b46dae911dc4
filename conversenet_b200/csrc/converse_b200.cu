// C ABI of the B200 Converse2D library: plan selection, kernel wrappers, launches.
// Declarations and the reference interfaces they replace are in include/converse_b200.h.
#include "../../include/converse_b200.h"
#include "cvb_internal.h"
#include "cvb_plan.h"
#include "cvb_block.cuh"
#include "cvb_rp_plan.h"

#include <algorithm>
#include <cstdlib>
#include <cstring>

namespace cvb {

static thread_local int g_last_cuda_error = 0;

int cuda_fail(cudaError_t e) {
  g_last_cuda_error = (int)e;
  return CVB_ERR_CUDA;
}

#ifdef CVB_TUNING
int env_int(const char* name, int dflt) {
  const char* v = getenv(name);
  return (v && *v) ? atoi(v) : dflt;
}
#endif

static int g_options[CVB_OPT_COUNT_] = {0, 0, 0, 3};
int option(int which) { return (which >= 0 && which < CVB_OPT_COUNT_) ? g_options[which] : 0; }

// generated by build.py: two launchers per compile-time plan
#define CVB_STATIC(a, b, c, d, nt, mb)                                                             \
  int launch_static_##a##_##b##_##c##_##d##_##nt##_##mb(const FwdParams&, int, size_t, int, cudaStream_t); \
  int launch_persist_##a##_##b##_##c##_##d##_##nt##_##mb(const FwdParams&, int, size_t, int, cudaStream_t);
#include "static_registry.inc"
#undef CVB_STATIC
static const StaticEntry kStatic[] = {
#define CVB_STATIC(a, b, c, d, nt, mb) \
  {a, b, c, d, nt, mb, launch_static_##a##_##b##_##c##_##d##_##nt##_##mb, launch_persist_##a##_##b##_##c##_##d##_##nt##_##mb},
#include "static_registry.inc"
#undef CVB_STATIC
};

// Device word set by a kernel whose bounded wait gave up (one per device).
__device__ int g_device_status;
int* status_ptr() {
  static int* ptrs[64] = {nullptr};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  if (!ptrs[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_device_status) != cudaSuccess) return nullptr;
    ptrs[dev] = (int*)p;
  }
  return ptrs[dev];
}

int sm_count() {
  static int n[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (!n[dev]) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
    n[dev] = v;
  }
  return n[dev];
}


// ------------------------------------------------------------------ kernels
// Tiled table build: one block per (channel, tile of table columns).
template <int CK, int CS>
__global__ void __launch_bounds__(256) transfer_tile_kernel(const TransferParams T) {
  __shared__ TransferTileSmem S;
  transfer_tile_block<CK, CS>(T, (long long)blockIdx.x, 0, S);
}

// Per-entry form: the twiddle and Rader tables behind the spectrum (first = C*h*w) and, for
// scales above kFastMaxScale, the whole table (first = 0).
__global__ void transfer_kernel(const TransferParams T, const size_t first) {
  const size_t total = (size_t)T.C * T.h * T.w;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const size_t n1 = total + T.h + T.w;
  const size_t n2 = n1 + (T.ry.R ? T.ry.R - 1 : 0);
  const size_t n3 = n2 + (T.rx.R ? T.rx.R - 1 : 0);
  for (size_t i = first + (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n3; i += stride) {
    if (i >= n2) {
      rader_entry(T, T.rx, (int)(i - n2));
    } else if (i >= n1) {
      rader_entry(T, T.ry, (int)(i - n1));
    } else if (i >= total) {
      twiddle_entry(T, (int)(i - total));
    } else {
      // posy fastest: matches the table's memory order
      const int posy = (int)(i % T.h);
      const size_t rest = i / T.h;
      const int posx = (int)(rest % T.w);
      const int c = (int)(rest / T.w);
      transfer_entry(T, c, posy, posx);
    }
  }
}

static int dispatch_smem(FwdParams& P, int io_dtype, cudaStream_t st) {
  const int esize = io_dtype == CVB_F32 ? 4 : 2;
  if (P.py.nst == 2 && P.px.nst == 2 && !option(CVB_OPT_RUNTIME_PLAN)) {
    // first registry line for this plan; CVB_VARIANT=n picks the n-th (tuning aid)
    int skip = CVB_TUNE("CVB_VARIANT", 0);
    for (const StaticEntry& e : kStatic) {
      if (!(e.ry0 == P.py.radix[0] && e.ry1 == P.py.radix[1] && e.rx0 == P.px.radix[0] &&
            e.rx1 == P.px.radix[1] && skip-- <= 0))
        continue;
      // Persistent blocks: a block loops over plane pairs and the raw planes of its next pair arrive by
      // bulk copies (TMA) into shared memory while the current pair is transformed.  Needs 16-byte
      // aligned planes, room for mb blocks per SM with the double buffer, and more pairs than blocks.
      // Default for bf16 tensors (the staged copy replaces the 2-byte global loads of the first column
      // stage: 37.8 us instead of 48.3 us on the 16 x 64 x 64 x 64 scale-2 layer); for fp32 it measured
      // 1-3 % slower than one block per pair, so there it is an option (CVB_OPT_PERSISTENT).
      const size_t psmem = persistent_smem_bytes(P.h, P.w, P.H, P.W, P.k, esize);
      const size_t plane_bytes = (size_t)P.H * P.W * esize;
      const int blocks = sm_count() * e.mb;
      const bool can_persist = plane_bytes % 16 == 0 && ((size_t)P.x) % 16 == 0 &&
                               psmem * e.mb <= kSmemLimit && num_pairs(P) > blocks &&
                               (option(CVB_OPT_PERSISTENT) != 0 || io_dtype == CVB_BF16);
      if (can_persist) {
        P.ystash = 0;
        return e.fn_persist(P, io_dtype, psmem, blocks, st);
      }
      return e.fn(P, io_dtype, smem_bytes_for(P.h, P.w, P.k, P.ystash), 0, st);
    }
  }
  return launch_dynamic(P, io_dtype, smem_bytes_for(P.h, P.w, P.k, P.ystash), st);
}

// true when the forward for this padded size takes the multi-pass path
static bool needs_strip(int h, int w, int k, bool big) {
  return big || smem_bytes_for(h, w, k) > kSmemLimit || option(CVB_OPT_MULTIPASS) != 0;
}

// chunk workspace of the multi-launch real-plane kernels
constexpr size_t kRpWorkspace = (size_t)64 << 20;

// Planes whose two lengths have a multi-pass pair plan that beats the real-plane kernels on FULL pairs of planes (two
// images of a batch share their taps and travel as one complex plane) have the tables of both kernel families:
//   tensor-core plans   268 and 516 (but see takes_contractions)
//   264 and 520         4 x 128 planes of 264 x 264: 280 us against 309, of 520 x 520: 1256 against 1463
//   dense stages that cost more than the two cheap butterflies of a three-stage plan (16 planes of n x n, one pair per
//   channel, real-plane kernels / pair kernels): 918 = 102 x 9 1.58, 1071 = 119 x 9 1.66, 1000 = 100 x 10 1.25,
//   1300 = 100 x 13 1.30, 891 = 81 x 11 1.14; but 1024 = 64 x 16 0.73, 1280 = 80 x 16 0.76, 900 = 60 x 15 0.88,
//   847 = 77 x 11 0.98.  Only on both axes (1000 x 1024: 1.01, 1000 x 720: 0.82), not with a large prime in the length
//   (776 = 97 x 8: 0.62), not for single planes (1000 x 1000, batch 1: 0.65)
// At scale >= 2 the run-time kernels' epilogue wins (260 x 260 by 2, 4 x 64 planes: 270 us against 596; 1071 x 1071 by 2,
// 2 x 8 planes: 1482 us against 1716).
static bool strip_axis(int n) { return n == 264 || n == 520; }
static bool three_stage_axis(int n) {
  int r0, r1;
  Plan1D pl;
  bool big = false;
  if (n <= 800 || !rp::axis_plan(n, r0, r1)) return false;
  const int width = rp::matrix_width(r0);
  return (width >= 56 || (width > 0 && r1 <= 11 && n > 860)) && make_plan(n, pl, &big) && !big;
}
static bool dual_tables(int h, int w) {
  return ((gemm_axis(h) && gemm_axis(w) && !gemm_disabled()) || (strip_axis(h) && strip_axis(w)) ||
          (three_stage_axis(h) && three_stage_axis(w))) && rp::supported(h, w);
}
static size_t dual_offset(int C, int h, int w) { return (rp::table_bytes(C, h, w) + 255) / 256 * 256; }
// Compile-time-plan kernels on pairs of planes that share their taps (k_static.cu), for the sizes that have one: with
// full pairs they beat the run-time plans (136 x 136, 4 x 128 planes: 53 us against 76; 68 x 68 upsampled by 2, 16 x 64
// planes: 37 against 42).  An odd batch leaves one pair half empty, which pays from five images on.
static bool static_plan(int h, int w) {
  for (const StaticEntry& e : kStatic)
    if (e.ry0 * e.ry1 == h && e.rx0 * e.rx1 == w) return true;
  return false;
}
static bool full_pairs(int B) { return B >= 2 && (B % 2 == 0 || B >= 5); }
static bool takes_static_pairs(int B, int h, int w) {
  return full_pairs(B) && !option(CVB_OPT_RUNTIME_PLAN) && !option(CVB_OPT_MULTIPASS) && static_plan(h, w) && rp::supported(h, w);
}
// (from seven images on where a full pair gains least: 1000 x 1000, 5 x 8 planes: 1755 us against 1661)
static bool takes_multipass_pairs(int B, int h, int w, int s) {
  return s == 1 && full_pairs(B) && dual_tables(h, w) && !(B == 5 && three_stage_axis(h));
}
// Of those, the ones that run on real planes all the same when the caller has the table for them: 268 x 268 (of the pair lengths
// the one that has integer contractions too), whose 67-point stages then keep a tenth of the rounding error (1.8e-7 against 2 to
// 4e-6 of the TF32 products).  Pairs / real planes, us: 2 x 32 planes 71 / 71, 2 x 48 133 / 133, 2 x 64 152 / 139, 2 x 96 204 / 209, 2 x 128
// 256 / 281, 8 x 128 971 / 1063: no slower up to 128 planes, up to 14 % slower above, which is the price of the accuracy.  From
// 128 planes on: smaller batches keep the one table that they always had.
static bool takes_contractions(int B, int C, int h, int w, int s) {
  return takes_multipass_pairs(B, h, w, s) && gemm_axis(h) && gemm_axis(w) && rp::fix_length(h) && rp::fix_length(w) &&
         (long long)B * C >= 128;
}

static int check_padding(int H, int W, int p, int pad_mode) {
  if (p < 0) return CVB_ERR_BAD_ARGUMENT;
  if (pad_mode < CVB_PAD_CIRCULAR || pad_mode > CVB_PAD_CONSTANT) return CVB_ERR_BAD_ARGUMENT;
  if (pad_mode == CVB_PAD_CIRCULAR && (p > H || p > W)) return CVB_ERR_BAD_PADDING;
  if (pad_mode == CVB_PAD_REFLECT && p > 0 && (p >= H || p >= W)) return CVB_ERR_BAD_PADDING;
  return CVB_OK;
}

}  // namespace cvb

using namespace cvb;

extern "C" {

int cvb_version(void) { return 100; }

const char* cvb_strerror(int status) {
  switch (status) {
    case CVB_OK: return "success";
    case CVB_ERR_BAD_ARGUMENT: return "bad argument (null pointer, non-positive size or unknown enum)";
    case CVB_ERR_BAD_PADDING: return "padding too wide for this padding_mode";
    case CVB_ERR_UNSUPPORTED_SIZE: return "padded plane size not supported by the FFT engine";
    case CVB_ERR_WORKSPACE: return "workspace missing or too small";
    case CVB_ERR_CUDA: return "CUDA runtime error (see cvb_last_cuda_error)";
    case CVB_ERR_KERNEL_TOO_LARGE: return "kernel_size larger than the padded plane";
    case CVB_ERR_TOO_LARGE: return "plane too large for the fixed scratch array of this entry point";
    default: return "unknown status";
  }
}

int cvb_last_cuda_error(void) { return g_last_cuda_error; }

int cvb_set_option(int which, int value) {
  if (which < 0 || which >= CVB_OPT_COUNT_) return CVB_ERR_BAD_ARGUMENT;
  if (which == CVB_OPT_BLOCK_KERNELS && (value < 0 || value > 3)) return CVB_ERR_BAD_ARGUMENT;
  g_options[which] = value;
  return CVB_OK;
}
int cvb_get_option(int which) { return (which >= 0 && which < CVB_OPT_COUNT_) ? g_options[which] : CVB_ERR_BAD_ARGUMENT; }

int cvb_last_device_status(int clear) {
  int* p = status_ptr();
  if (!p) return CVB_ERR_CUDA;
  int v = 0;
  CVB_CUDA(cudaDeviceSynchronize());
  CVB_CUDA(cudaMemcpy(&v, p, sizeof(int), cudaMemcpyDeviceToHost));
  if (clear && v) {
    const int zero = 0;
    CVB_CUDA(cudaMemcpy(p, &zero, sizeof(int), cudaMemcpyHostToDevice));
  }
  return v;
}

int cvb_plan_radices(int n, int* radices, int max_stages) {
  Plan1D pl;
  if (!make_plan(n, pl)) return 0;
  if (radices)
    for (int i = 0; i < pl.nst && i < max_stages; ++i) radices[i] = pl.radix[i];
  return pl.nst;
}

int cvb_fits_shared(int h, int w) {
  if (h < 2 || w < 2) return CVB_ERR_BAD_ARGUMENT;
  Plan1D py, px;
  bool big = false;
  if (!make_axis_plans(h, w, py, px, &big)) return CVB_ERR_UNSUPPORTED_SIZE;
  return needs_strip(h, w, kMaxTaps, big) ? 0 : 1;
}

static size_t pair_table_bytes(int C, int h, int w) {
  Plan1D py, px;
  // sized for the register-FFT plans (with their Rader tables) where they exist, so that the size
  // does not depend on which multi-pass kernels serve the plane
  if (!make_plan(h, py) || !make_plan(w, px)) {
    if (!make_axis_plans(h, w, py, px)) return 0;
  }
  RaderInfo ry, rx;
  rader_both(py, px, ry, rx);
  return ((size_t)C * h * w + h + w + rader_blob_float2(ry) + rader_blob_float2(rx)) * sizeof(float2);
}

// The real-plane table alone, the pair table alone (lengths without a two-stage plan), or one behind the other (sizes with
// dual_tables).  Sizes of k_static.cu read the real-plane table in a blob that keeps the pair table's size, which callers
// have allocated since before there were two.
size_t cvb_transfer_bytes(int C, int h, int w) {
  if (C < 1 || h < 2 || w < 2) return 0;
  const size_t plane = rp::table_bytes(C, h, w);
  if (plane && !dual_tables(h, w) && !static_plan(h, w)) return plane;
  const size_t n = pair_table_bytes(C, h, w);
  return n == 0 ? 0 : plane && dual_tables(h, w) ? n + dual_offset(C, h, w) : std::max(n, plane);
}
size_t cvb_pair_transfer_bytes(int C, int h, int w) { return C < 1 || h < 2 || w < 2 ? 0 : pair_table_bytes(C, h, w); }
size_t cvb_plane_transfer_bytes(int C, int h, int w) { return C < 1 || h < 2 || w < 2 ? 0 : rp::table_bytes(C, h, w); }

int cvb_takes_pairs(int B, int h, int w, int s) {
  return takes_multipass_pairs(B, h, w, s) ? 2 : takes_static_pairs(B, h, w) ? 1 : 0;
}

enum Tables { kAnyBatch, kPairTable, kPlaneTable };
static int build_table(const float* weight, const float* bias, int C, int k, int s, int h, int w, float eps,
                       int kind, void* table, void* stream, Tables which = kAnyBatch);
int cvb_build_pair_transfer(const float* weight, const float* bias, int C, int k, int s, int h, int w, float eps,
                            void* table, void* stream) {
  return build_table(weight, bias, C, k, s, h, w, eps, 0, table, stream, kPairTable);
}
int cvb_build_plane_transfer(const float* weight, const float* bias, int C, int k, int s, int h, int w, float eps,
                             void* table, void* stream) {
  return build_table(weight, bias, C, k, s, h, w, eps, 0, table, stream, kPlaneTable);
}

int cvb_build_transfer(const float* weight, const float* bias, int C, int k, int s, int h, int w,
                       float eps, void* table, void* stream) {
  return build_table(weight, bias, C, k, s, h, w, eps, 0, table, stream);
}

int cvb_build_x0_table(const float* weight, const float* bias, int C, int k, int s, int h, int w,
                       float eps, void* table, void* stream) {
  return build_table(weight, bias, C, k, s, h, w, eps, 1, table, stream);
}

static int build_table(const float* weight, const float* bias, int C, int k, int s, int h, int w, float eps,
                       int kind, void* table, void* stream, Tables which) {
  if (!weight || !bias || !table || C < 1 || k < 1 || s < 1 || h < 2 || w < 2) return CVB_ERR_BAD_ARGUMENT;
  // the tiled build keeps k-long arrays of kMaxTaps entries per thread and per block
  if (k > kMaxTaps || k > s * h || k > s * w) return CVB_ERR_KERNEL_TOO_LARGE;
  if (which != kPairTable && rp::supported(h, w)) {
    const int rc = rp::build_table(weight, bias, C, k, s, h, w, eps, kind, table, (cudaStream_t)stream);
    if (rc != CVB_OK || which == kPlaneTable || !dual_tables(h, w)) return rc;
    table = (char*)table + dual_offset(C, h, w);
  }
  if (which == kPlaneTable) return CVB_ERR_UNSUPPORTED_SIZE;
  TransferParams T;
  if (!make_axis_plans(h, w, T.py, T.px)) return CVB_ERR_UNSUPPORTED_SIZE;
  T.weight = weight; T.bias = bias; T.table = (float2*)table;
  T.C = C; T.k = k; T.s = s; T.h = h; T.w = w; T.eps = eps; T.kind = kind;
  rader_both(T.py, T.px, T.ry, T.rx);
  const size_t total = (size_t)C * h * w + h + w + rader_blob_float2(T.ry) + rader_blob_float2(T.rx);
  const size_t spectrum = (size_t)C * h * w;
  size_t first = 0;
  if (s <= kFastMaxScale) {
    const long long nblk = (long long)C * ((w + kTransferTile - 1) / kTransferTile);
    if (nblk > 0x7fffffffLL) return CVB_ERR_TOO_LARGE;
    cudaStream_t st = (cudaStream_t)stream;
    switch (k * 10 + s) {
#define X(KK, SS) \
      case KK * 10 + SS: transfer_tile_kernel<KK, SS><<<(int)nblk, 256, 0, st>>>(T); break;
      CVB_TRANSFER_CASES(X)
#undef X
      default: transfer_tile_kernel<0, 0><<<(int)nblk, 256, 0, st>>>(T); break;
    }
    CVB_CUDA(cudaGetLastError());
    first = spectrum;
  }
  const int threads = 128;
  const int blocks = (int)std::min<size_t>((total - first + threads - 1) / threads, 148 * 64);
  transfer_kernel<<<blocks, threads, 0, (cudaStream_t)stream>>>(T, first);
  CVB_CUDA(cudaGetLastError());
  return CVB_OK;
}

static size_t pair_workspace(int B, int C, int h, int w, int s) {
  Plan1D py, px;
  bool big = false;
  if (h < 2 || w < 2 || (static_plan(h, w) && !option(CVB_OPT_MULTIPASS)) || !make_axis_plans(h, w, py, px, &big)) return 0;
  if (!needs_strip(h, w, kMaxTaps, big)) return 0;
  return strip_geometry(h, w, kMaxTaps, s, C * ((B + 1) / 2)).ws_bytes;
}

// The kernels that carry two planes with the same taps as one complex plane.  hh: the table's form (FwdParams::hh).
static int pair_forward(const void* x, void* out, const void* table, const float* weight, int B, int C, int H, int W, int k,
                        int s, int p, int pad_mode, int io_dtype, int fuse_gelu, int hh, void* workspace,
                        size_t workspace_bytes, cudaStream_t st) {
  FwdParams P;
  P.x = x; P.out = out; P.table = (const float2*)table; P.weight = weight;
  P.B = B; P.C = C; P.H = H; P.W = W; P.k = k; P.s = s; P.p = p; P.pad_mode = pad_mode;
  P.fuse_gelu = fuse_gelu ? 1 : 0;
  P.h = H + 2 * p; P.w = W + 2 * p; P.pitch = P.w | 1;
  P.hh = hh;
  P.skip_mask = CVB_TUNE("CVB_SKIP", 0);
  P.status = status_ptr();
  P.ystash = CVB_TUNE("CVB_NO_YSTASH", 0) ? 0 : choose_ystash(P.h, P.w, k, s);
  bool big = false;
  if (!make_axis_plans(P.h, P.w, P.py, P.px, &big)) return CVB_ERR_UNSUPPORTED_SIZE;
  // workspace need is computed with the largest tap count so that it does not depend on k
  if (needs_strip(P.h, P.w, kMaxTaps, big)) {
    P.ystash = 0;
    return launch_strip(P, io_dtype, workspace, workspace_bytes, st);
  }
  return dispatch_smem(P, io_dtype, st);
}

static int check_forward(const void* x, void* out, const void* table, const float* weight, int B, int C, int H, int W, int k,
                         int s, int p, int pad_mode, int io_dtype) {
  if (!x || !out || !table || B < 1 || C < 1 || H < 1 || W < 1 || k < 1 || s < 1) return CVB_ERR_BAD_ARGUMENT;
  if (s > 1 && !weight) return CVB_ERR_BAD_ARGUMENT;
  if (io_dtype != CVB_F32 && io_dtype != CVB_BF16) return CVB_ERR_BAD_ARGUMENT;
  if (k > kMaxTaps) return CVB_ERR_KERNEL_TOO_LARGE;
  const int rc = check_padding(H, W, p, pad_mode);
  if (rc != CVB_OK) return rc;
  if (H + 2 * p < 2 || W + 2 * p < 2) return CVB_ERR_BAD_ARGUMENT;
  return k > s * (H + 2 * p) || k > s * (W + 2 * p) ? CVB_ERR_KERNEL_TOO_LARGE : CVB_OK;
}

int cvb_pair_fwd(const void* x, void* out, const void* table, const float* weight, int B, int C, int H, int W, int k, int s,
                 int p, int pad_mode, int io_dtype, int fuse_gelu, void* workspace, size_t workspace_bytes, void* stream) {
  const int rc = check_forward(x, out, table, weight, B, C, H, W, k, s, p, pad_mode, io_dtype);
  if (rc != CVB_OK) return rc;
  return pair_forward(x, out, table, weight, B, C, H, W, k, s, p, pad_mode, io_dtype, fuse_gelu, 0, workspace,
                      workspace_bytes, (cudaStream_t)stream);
}

static rp::Route plane_route(int B, int C, int H, int W, int s, int p) {
  return rp::route(B, C, H, W, s, p, sm_count(), option(CVB_OPT_MULTIPASS) != 0,
                   std::max(kRpWorkspace, rp::ws_plane_bytes(H + 2 * p, W + 2 * p, s)));
}

size_t cvb_converse2d_workspace_bytes(int B, int C, int H, int W, int s, int p, int io_dtype) {
  (void)io_dtype;
  if (B < 1 || C < 1 || H < 1 || W < 1 || p < 0 || s < 1) return 0;
  const int h = H + 2 * p, w = W + 2 * p;
  if (takes_static_pairs(B, h, w)) return 0;
  if (rp::supported(h, w) && !takes_multipass_pairs(B, h, w, s))
    return plane_route(B, C, H, W, s, p).ws_bytes;
  return pair_workspace(B, C, h, w, s);
}
size_t cvb_pair_workspace_bytes(int B, int C, int H, int W, int s, int p) {
  if (B < 1 || C < 1 || H < 1 || W < 1 || p < 0 || s < 1) return 0;
  return pair_workspace(B, C, H + 2 * p, W + 2 * p, s);
}

int cvb_takes_planes(int B, int C, int h, int w, int s) {
  return B > 0 && C > 0 && h > 1 && w > 1 && s > 0 && takes_contractions(B, C, h, w, s) ? 1 : 0;
}
size_t cvb_plane_workspace_bytes(int B, int C, int H, int W, int s, int p) {
  if (B < 1 || C < 1 || H < 1 || W < 1 || p < 0 || s < 1 || !rp::supported(H + 2 * p, W + 2 * p)) return 0;
  return plane_route(B, C, H, W, s, p).ws_bytes;
}
int cvb_plane_fwd(const void* x, void* out, const void* table, const float* weight, int B, int C, int H, int W, int k, int s,
                  int p, int pad_mode, int io_dtype, int fuse_gelu, void* workspace, size_t workspace_bytes, void* stream) {
  const int rc = check_forward(x, out, table, weight, B, C, H, W, k, s, p, pad_mode, io_dtype);
  if (rc != CVB_OK) return rc;
  rp::Params Q;
  if (!rp::fill_params(Q, table, B, C, H, W, k, s, p, pad_mode)) return CVB_ERR_UNSUPPORTED_SIZE;
  Q.x = x; Q.out = out; Q.weight = weight; Q.gelu = fuse_gelu ? 1 : 0;
  return rp::run(Q, plane_route(B, C, H, W, s, p), io_dtype, workspace, workspace_bytes, (cudaStream_t)stream);
}

int cvb_converse2d_fwd(const void* x, void* out, const void* table, const float* weight, int B,
                       int C, int H, int W, int k, int s, int p, int pad_mode, int io_dtype,
                       int fuse_gelu, void* workspace, size_t workspace_bytes, void* stream) {
  const int rc = check_forward(x, out, table, weight, B, C, H, W, k, s, p, pad_mode, io_dtype);
  if (rc != CVB_OK) return rc;
  const int h = H + 2 * p, w = W + 2 * p;
  int hh = 0;
  rp::Params Q;
  if (takes_multipass_pairs(B, h, w, s)) {
    table = (const char*)table + dual_offset(C, h, w);
  } else if (takes_static_pairs(B, h, w)) {
    hh = h / 2 + 1;
  } else if (rp::fill_params(Q, table, B, C, H, W, k, s, p, pad_mode)) {
    Q.x = x; Q.out = out; Q.weight = weight; Q.gelu = fuse_gelu ? 1 : 0;
    return rp::run(Q, plane_route(B, C, H, W, s, p), io_dtype, workspace, workspace_bytes, (cudaStream_t)stream);
  }
  return pair_forward(x, out, table, weight, B, C, H, W, k, s, p, pad_mode, io_dtype, fuse_gelu, hh, workspace,
                      workspace_bytes, (cudaStream_t)stream);
}

int cvb_cross_spectrum_supported(int h, int w) {
  if (h < 2 || w < 2) return CVB_ERR_BAD_ARGUMENT;
  Plan1D py, px;
  if (!make_plan(h, py) || !make_plan(w, px)) return 0;
  if (plan_has_big(py) || plan_has_big(px)) return 0;
  return xspec_smem_bytes(h, w, 0) <= kSmemLimit ? 1 : xspec_smem_bytes(h, w, 1) <= kSmemLimit ? 2 : 0;
}

int cvb_cross_spectrum(const float* x, const float* q, const void* table, void* out, int nseg, int B, int C,
                       int H, int W, int p, int pad_mode, void* stream) {
  if (!x || !q || !table || !out || nseg < 1 || B < 1 || C < 1 || H < 1 || W < 1) return CVB_ERR_BAD_ARGUMENT;
  if (nseg > B || nseg > 65535) return CVB_ERR_BAD_ARGUMENT;
  const int rc = check_padding(H, W, p, pad_mode);
  if (rc != CVB_OK) return rc;
  XspecParams Q;
  Q.x = x; Q.q = q; Q.out = (float2*)out;
  Q.B = B; Q.C = C; Q.H = H; Q.W = W; Q.p = p; Q.pad_mode = pad_mode;
  Q.h = H + 2 * p; Q.w = W + 2 * p; Q.pitch = Q.w | 1; Q.nseg = nseg;
  if (Q.h < 2 || Q.w < 2) return CVB_ERR_BAD_ARGUMENT;
  const int kind = cvb_cross_spectrum_supported(Q.h, Q.w);
  if (kind != 1 && kind != 2) return CVB_ERR_UNSUPPORTED_SIZE;
  Q.direct = kind == 2 ? 1 : 0;
  if (!make_plan(Q.h, Q.py) || !make_plan(Q.w, Q.px)) return CVB_ERR_UNSUPPORTED_SIZE;
  // the twiddles behind the multiplier
  Q.tw = (const float2*)table + (rp::supported(Q.h, Q.w) ? (size_t)C * Q.w * (Q.h / 2 + 1) : (size_t)C * Q.h * Q.w);
  return launch_xspec(Q, (cudaStream_t)stream);
}

int cvb_tap_gradient(const float* g_full, const float* r, float* out, int nseg, int B, int C, int h, int w, int k,
                     int s, void* stream) {
  if (!g_full || !r || !out || nseg < 1 || B < 1 || C < 1 || h < 1 || w < 1 || k < 1 || s < 1) return CVB_ERR_BAD_ARGUMENT;
  if (nseg > B || nseg > 65535) return CVB_ERR_BAD_ARGUMENT;
  if (k > s * h || k > s * w) return CVB_ERR_KERNEL_TOO_LARGE;
  return launch_tap_gradient(g_full, r, out, nseg, B, C, h, w, k, s, (cudaStream_t)stream);
}

// Allocation-free variant: always the multi-pass kernels, scratch = the library's fixed
// device array (see k_strip.cu).  Own copy of the argument checks so that the entry
// point above stays as it is.
int cvb_converse2d_fwd_static_scratch(const void* x, void* out, const void* table, const float* weight,
                                      int B, int C, int H, int W, int k, int s, int p, int pad_mode,
                                      int io_dtype, int fuse_gelu, void* stream) {
  if (!x || !out || !table || B < 1 || C < 1 || H < 1 || W < 1 || k < 1 || s < 1) return CVB_ERR_BAD_ARGUMENT;
  if (s > 1 && !weight) return CVB_ERR_BAD_ARGUMENT;
  if (io_dtype != CVB_F32 && io_dtype != CVB_BF16) return CVB_ERR_BAD_ARGUMENT;
  if (k > kMaxTaps) return CVB_ERR_KERNEL_TOO_LARGE;
  const int rc = check_padding(H, W, p, pad_mode);
  if (rc != CVB_OK) return rc;
  rp::Params Q;
  if (k <= s * (H + 2 * p) && k <= s * (W + 2 * p) && rp::fill_params(Q, table, B, C, H, W, k, s, p, pad_mode)) {
    if ((size_t)Q.h * Q.w * sizeof(float2) > CVB_STATIC_SCRATCH_BYTES) return CVB_ERR_TOO_LARGE;
    Q.x = x; Q.out = out; Q.weight = weight; Q.gelu = fuse_gelu ? 1 : 0;
    void* scratch = nullptr;
    const int rs = static_scratch_address(&scratch);
    if (rs != CVB_OK) return rs;
    return rp::run(Q, rp::route(B, C, H, W, s, p, sm_count(), true, CVB_STATIC_SCRATCH_BYTES), io_dtype, scratch,
                   CVB_STATIC_SCRATCH_BYTES, (cudaStream_t)stream);
  }
  FwdParams P;
  P.x = x; P.out = out; P.table = (const float2*)table; P.weight = weight;
  P.B = B; P.C = C; P.H = H; P.W = W; P.k = k; P.s = s; P.p = p; P.pad_mode = pad_mode;
  P.fuse_gelu = fuse_gelu ? 1 : 0;
  P.h = H + 2 * p; P.w = W + 2 * p; P.pitch = P.w | 1;
  P.skip_mask = 0;
  P.status = status_ptr();  // an address look-up cached per device, no allocation
  P.ystash = 0;
  if (P.h < 2 || P.w < 2) return CVB_ERR_BAD_ARGUMENT;
  if (k > s * P.h || k > s * P.w) return CVB_ERR_KERNEL_TOO_LARGE;
  if (!make_axis_plans(P.h, P.w, P.py, P.px)) return CVB_ERR_UNSUPPORTED_SIZE;
  if ((size_t)P.h * P.w * sizeof(float2) > CVB_STATIC_SCRATCH_BYTES) return CVB_ERR_TOO_LARGE;
  return launch_strip_static_scratch(P, io_dtype, (cudaStream_t)stream);
}

int cvb_ln_pw_gelu_fwd(const void* x, void* out, const float* ln_w, const float* ln_b, float ln_eps,
                       const float* w, const float* b, int B, int C, int HW, int io_dtype, void* stream) {
  if (!x || !out || !ln_w || !ln_b || !w || !b || B < 1 || HW < 1) return CVB_ERR_BAD_ARGUMENT;
  if (io_dtype != CVB_F32 && io_dtype != CVB_BF16) return CVB_ERR_BAD_ARGUMENT;
  if (C != kBlkC) return CVB_ERR_UNSUPPORTED_SIZE;
  BlockParams P;
  memset(&P, 0, sizeof(P));
  P.x = x; P.out = out; P.ln_w = ln_w; P.ln_b = ln_b; P.ln_eps = ln_eps; P.w_a = w; P.b_a = b;
  P.B = B; P.HW = HW;
  // tensor-core path (tcgen05): fp32 tensors whose images are whole 128-pixel tiles, 16-byte aligned;
  // option CVB_OPT_BLOCK_KERNELS: 0 forces the CUDA-core kernel, 1 the single-buffered tensor-core
  // kernel, 2 the warp-specialised one with operand tiles in shared memory, 3 (default) the one that
  // streams the tensors through a cp.async ring and stages the operand in tensor memory
  // (the single-buffered kernel is fp32 only; bf16 tensors take a warp-specialised one)
  const int bk = option(CVB_OPT_BLOCK_KERNELS);
  if (bk && HW % 128 == 0 && ((size_t)x) % 16 == 0 && (io_dtype == CVB_F32 || bk >= 2))
    return bk == 3   ? launch_ln_pw_gelu_tc3(P, io_dtype, sm_count(), status_ptr(), (cudaStream_t)stream)
           : bk == 2 ? launch_ln_pw_gelu_tc2(P, io_dtype, sm_count(), status_ptr(), (cudaStream_t)stream)
                     : launch_ln_pw_gelu_tc(P, sm_count(), status_ptr(), (cudaStream_t)stream);
  return launch_ln_pw_gelu(P, io_dtype, (cudaStream_t)stream);
}

int cvb_pw_res_mlp_fwd(const void* t, const void* x, void* out, const float* w2, const float* b2,
                       const float* alpha1, const float* ln_w, const float* ln_b, float ln_eps,
                       const float* w3, const float* b3, const float* w4, const float* b4,
                       const float* alpha2, int B, int C, int HW, int io_dtype, void* stream) {
  if (!t || !x || !out || !w2 || !b2 || !ln_w || !ln_b || !w3 || !b3 || !w4 || !b4 || B < 1 || HW < 1)
    return CVB_ERR_BAD_ARGUMENT;
  if (io_dtype != CVB_F32 && io_dtype != CVB_BF16) return CVB_ERR_BAD_ARGUMENT;
  if (C != kBlkC) return CVB_ERR_UNSUPPORTED_SIZE;
  BlockParams P;
  memset(&P, 0, sizeof(P));
  P.t = t; P.x = x; P.out = out; P.ln_w = ln_w; P.ln_b = ln_b; P.ln_eps = ln_eps;
  P.w_a = w2; P.b_a = b2; P.w_b = w3; P.b_b = b3; P.w_c = w4; P.b_c = b4;
  P.alpha1 = alpha1; P.alpha2 = alpha2;
  P.B = B; P.HW = HW;
  return launch_pw_res_mlp(P, io_dtype, sm_count(), (cudaStream_t)stream);
}

int cvb_pw_res_fwd(const void* t, const void* res, void* out, const float* w, const float* b,
                   const float* alpha, int B, int C, int HW, int io_dtype, void* stream) {
  if (!t || !res || !out || !w || !b || B < 1 || HW < 1) return CVB_ERR_BAD_ARGUMENT;
  if (io_dtype != CVB_F32 && io_dtype != CVB_BF16) return CVB_ERR_BAD_ARGUMENT;
  if (C != kBlkC || HW % 128 != 0 || ((size_t)t) % 16 != 0) return CVB_ERR_UNSUPPORTED_SIZE;
  if (io_dtype == CVB_BF16 && option(CVB_OPT_BLOCK_KERNELS) == 1) return CVB_ERR_UNSUPPORTED_SIZE;
  BlockParams P;
  memset(&P, 0, sizeof(P));
  P.t = t; P.x = res; P.out = out; P.w_a = w; P.b_a = b; P.alpha1 = alpha; P.B = B; P.HW = HW;
  const int bk = option(CVB_OPT_BLOCK_KERNELS);
  return bk == 3   ? launch_pw_res_tc3(P, io_dtype, sm_count(), status_ptr(), (cudaStream_t)stream)
         : bk != 1 ? launch_pw_res_tc2(P, io_dtype, sm_count(), status_ptr(), (cudaStream_t)stream)
                   : launch_pw_res_tc(P, sm_count(), status_ptr(), (cudaStream_t)stream);
}

int cvb_converse2d_fwd_train(const void* x, void* out, const void* table, const float* weight, float* r_keep, int B,
                             int C, int H, int W, int k, int s, int p, int pad_mode, int io_dtype, void* workspace,
                             size_t workspace_bytes, void* stream) {
  if (!x || !out || !table || B < 1 || C < 1 || H < 1 || W < 1 || k < 1 || s < 1) return CVB_ERR_BAD_ARGUMENT;
  if (s > 1 && !weight) return CVB_ERR_BAD_ARGUMENT;
  if (io_dtype != CVB_F32 && io_dtype != CVB_BF16) return CVB_ERR_BAD_ARGUMENT;
  if (k > kMaxTaps || k > s * (H + 2 * p) || k > s * (W + 2 * p)) return CVB_ERR_KERNEL_TOO_LARGE;
  const int rc = check_padding(H, W, p, pad_mode);
  if (rc != CVB_OK) return rc;
  if (H + 2 * p < 2 || W + 2 * p < 2 || !rp::supported(H + 2 * p, W + 2 * p)) return CVB_ERR_UNSUPPORTED_SIZE;
  if (s == 1)    // nothing to keep
    return cvb_converse2d_fwd(x, out, table, weight, B, C, H, W, k, s, p, pad_mode, io_dtype, 0, workspace, workspace_bytes,
                              stream);
  rp::Params Q;
  rp::fill_params(Q, table, B, C, H, W, k, s, p, pad_mode);
  if (takes_static_pairs(B, Q.h, Q.w)) {
    FwdParams P;
    if (!make_axis_plans(Q.h, Q.w, P.py, P.px)) return CVB_ERR_UNSUPPORTED_SIZE;
    P.x = x; P.out = out; P.table = (const float2*)table; P.weight = weight;
    P.B = B; P.C = C; P.H = H; P.W = W; P.k = k; P.s = s; P.p = p; P.pad_mode = pad_mode; P.fuse_gelu = 0;
    P.h = Q.h; P.w = Q.w; P.pitch = P.w | 1; P.hh = Q.hh; P.skip_mask = 0; P.status = status_ptr();
    P.ystash = choose_ystash(P.h, P.w, k, s);
    P.rsave = r_keep;
    return dispatch_smem(P, io_dtype, (cudaStream_t)stream);
  }
  Q.x = x; Q.out = out; Q.weight = weight; Q.rsave = r_keep;
  const rp::Route r = rp::route(B, C, H, W, s, p, sm_count(), option(CVB_OPT_MULTIPASS) != 0,
                                std::max(kRpWorkspace, rp::ws_plane_bytes(Q.h, Q.w, s)));
  return rp::run(Q, r, io_dtype, workspace, workspace_bytes, (cudaStream_t)stream);
}

size_t cvb_converse2d_train_workspace_bytes(int B, int C, int H, int W, int s, int p) {
  if (B < 1 || C < 1 || H < 1 || W < 1 || p < 0 || s < 1 || !rp::supported(H + 2 * p, W + 2 * p)) return 0;
  if (s == 1) return cvb_converse2d_workspace_bytes(B, C, H, W, s, p, CVB_F32);
  if (takes_static_pairs(B, H + 2 * p, W + 2 * p)) return 0;
  return rp::route(B, C, H, W, s, p, sm_count(), option(CVB_OPT_MULTIPASS) != 0,
                   std::max(kRpWorkspace, rp::ws_plane_bytes(H + 2 * p, W + 2 * p, s))).ws_bytes;
}

size_t cvb_converse2d_bwd_workspace_bytes(int B, int C, int H, int W, int k, int s, int p, int want_x, int want_params) {
  if (B < 1 || C < 1 || H < 1 || W < 1 || k < 1 || k > kMaxTaps || p < 0 || s < 1) return 0;
  if (!rp::supported(H + 2 * p, W + 2 * p)) return 0;
  return rp::bwd_workspace(B, C, H, W, k, s, p, want_x != 0, want_params != 0, sm_count());
}

int cvb_converse2d_bwd(const float* x, const float* g, const float* r, const void* table, const float* weight,
                       const float* bias, float* gx, float* gw, float* gb, int B, int C, int H, int W, int k, int s,
                       int p, int pad_mode, float eps, void* workspace, size_t workspace_bytes, void* stream) {
  if (!g || !table || !weight || B < 1 || C < 1 || H < 1 || W < 1 || k < 1 || s < 1) return CVB_ERR_BAD_ARGUMENT;
  if ((gw == nullptr) != (gb == nullptr) || (!gx && !gw)) return CVB_ERR_BAD_ARGUMENT;
  if (gw && (!x || !bias)) return CVB_ERR_BAD_ARGUMENT;
  if (k > kMaxTaps || k > s * (H + 2 * p) || k > s * (W + 2 * p)) return CVB_ERR_KERNEL_TOO_LARGE;
  const int rc = check_padding(H, W, p, pad_mode);
  if (rc != CVB_OK) return rc;
  return rp::run_bwd(x, g, r, table, weight, bias, gx, gw, gb, B, C, H, W, k, s, p, pad_mode, eps, workspace,
                     workspace_bytes, sm_count(), (cudaStream_t)stream);
}

int cvb_block_pre_train(const float* x, float* out, float* z1, const void* pack, float ln_eps, int B, int HW,
                        void* stream) {
  if (!x || !out || !z1 || !pack || ((size_t)pack) % 16 || B < 1 || HW < 1) return CVB_ERR_BAD_ARGUMENT;
  return launch_block_mix_train(false, x, nullptr, out, z1, nullptr, pack, ln_eps, B, HW, sm_count(), status_ptr(),
                                (cudaStream_t)stream);
}

int cvb_block_post_train(const float* u, const float* x, float* out, float* x1, float* z3, const void* pack, float ln_eps,
                         int B, int HW, void* stream) {
  if (!u || !x || !out || !x1 || !z3 || !pack || ((size_t)pack) % 16 || B < 1 || HW < 1) return CVB_ERR_BAD_ARGUMENT;
  return launch_block_mix_train(true, x, u, out, z3, x1, pack, ln_eps, B, HW, sm_count(), status_ptr(),
                                (cudaStream_t)stream);
}

size_t cvb_block_grad_floats(void) { return block_grad_floats(); }

size_t cvb_block_bwd_workspace_bytes(int B, int H, int W, int k, int p) {
  const size_t conv = cvb_converse2d_bwd_workspace_bytes(B, kBlkM, H, W, k, 1, p, 1, 1);
  return conv ? block_grad_workspace(B, H * W, conv, sm_count()) : 0;
}

int cvb_block_bwd(const cvb_block_bwd_args* args) {
  if (!args) return CVB_ERR_BAD_ARGUMENT;
  const cvb_block_bwd_args& A = *args;
  const void* need[] = {A.x, A.t1, A.z1, A.u, A.x1, A.z3, A.g, A.table, A.conv_w, A.conv_b, A.ln1_w, A.ln1_b, A.w1, A.b1,
                        A.w2, A.b2, A.ln2_w, A.ln2_b, A.w3, A.b3, A.w4, A.b4, A.gx, A.gconv_w, A.gconv_b, A.gparams};
  for (const void* q : need)
    if (!q) return CVB_ERR_BAD_ARGUMENT;
  if (A.B < 1 || A.H < 1 || A.W < 1) return CVB_ERR_BAD_ARGUMENT;
  const int rc = check_padding(A.H, A.W, A.p, A.pad_mode);
  if (rc != CVB_OK) return rc;
  const size_t conv = cvb_converse2d_bwd_workspace_bytes(A.B, kBlkM, A.H, A.W, A.k, 1, A.p, 1, 1);
  if (!conv) return CVB_ERR_UNSUPPORTED_SIZE;
  return run_block_grad(A, conv, sm_count(), status_ptr(), (cudaStream_t)A.stream,
                        [](const cvb_block_bwd_args& a, const float* gu, float* gt, void* ws, size_t bytes) {
                          return rp::run_bwd(a.t1, gu, nullptr, a.table, a.conv_w, a.conv_b, gt, a.gconv_w, a.gconv_b, a.B,
                                             kBlkM, a.H, a.W, a.k, 1, a.p, a.pad_mode, a.conv_eps, ws, bytes, sm_count(),
                                             (cudaStream_t)a.stream);
                        });
}

size_t cvb_block_pack_bytes(void) { return block_pack_bytes(); }

int cvb_block_pack(const float* ln1_w, const float* ln1_b, const float* w1, const float* b1, const float* w2,
                   const float* b2, const float* alpha1, const float* ln2_w, const float* ln2_b, const float* w3,
                   const float* b3, const float* w4, const float* b4, const float* alpha2, void* pack, void* stream) {
  if (!ln1_w || !ln1_b || !w1 || !b1 || !w2 || !b2 || !ln2_w || !ln2_b || !w3 || !b3 || !w4 || !b4 || !pack)
    return CVB_ERR_BAD_ARGUMENT;
  return launch_block_pack(ln1_w, ln1_b, w1, b1, w2, b2, alpha1, ln2_w, ln2_b, w3, b3, w4, b4, alpha2, pack,
                           (cudaStream_t)stream);
}

int cvb_block_pre_fwd(const void* x, void* out, const void* pack, float ln_eps, int B, int HW, int io_dtype,
                      void* stream) {
  if (!x || !out || !pack || ((size_t)pack) % 16 || B < 1 || HW < 1) return CVB_ERR_BAD_ARGUMENT;
  if (io_dtype != CVB_F32 && io_dtype != CVB_BF16) return CVB_ERR_BAD_ARGUMENT;
  return launch_block_mix(false, x, nullptr, out, pack, ln_eps, B, HW, io_dtype, sm_count(), status_ptr(),
                          (cudaStream_t)stream);
}

int cvb_block_post_fwd(const void* t, const void* x, void* out, const void* pack, float ln_eps, int B, int HW,
                       int io_dtype, void* stream) {
  if (!t || !x || !out || !pack || ((size_t)pack) % 16 || B < 1 || HW < 1) return CVB_ERR_BAD_ARGUMENT;
  if (io_dtype != CVB_F32 && io_dtype != CVB_BF16) return CVB_ERR_BAD_ARGUMENT;
  return launch_block_mix(true, x, t, out, pack, ln_eps, B, HW, io_dtype, sm_count(), status_ptr(),
                          (cudaStream_t)stream);
}

}  // extern "C"
