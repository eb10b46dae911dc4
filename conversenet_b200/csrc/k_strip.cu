// Multi-pass (strip) kernels for planes that do not fit in shared memory: three
// launches per chunk of plane pairs, meeting in the caller's workspace.
#include <algorithm>
#include "../../include/converse_b200.h"
#include "cvb_internal.h"
#include "cvb_strip2.cuh"
#include "cvb_gemmdft.cuh"
#include "cvb_plan.h"

namespace cvb {

// generated by build.py: launchers of the compile-time axis plans
#define CVB_STRIP2(a, b, c, d)                                                    \
  int launch_strip2A_##a##_##b(const StripParams&, int, cudaStream_t);            \
  int launch_strip2B_##a##_##b(const StripParams&, int, cudaStream_t);            \
  int launch_strip2C_##a##_##b(const StripParams&, int, cudaStream_t);            \
  int launch_strip2Q_##a##_##b(int, int, int*);
#include "strip2_registry.inc"
#undef CVB_STRIP2
static const Strip2Entry kStrip2[] = {
#define CVB_STRIP2(a, b, c, d) {a, b, c, d, launch_strip2A_##a##_##b, launch_strip2B_##a##_##b, launch_strip2C_##a##_##b, launch_strip2Q_##a##_##b},
#include "strip2_registry.inc"
#undef CVB_STRIP2
};

static const Strip2Entry* find_strip2(const Plan1D& pl, const RaderInfo& ri) {
  if (pl.nst != 2) return nullptr;
  for (const Strip2Entry& e : kStrip2) {
    if (e.r0 != pl.radix[0] || e.r1 != pl.radix[1]) continue;
    if (e.s0 == 0) return &e;
    if (ri.R == e.r0 && ri.sub.nst == 2 && ri.sub.radix[0] == e.s0 && ri.sub.radix[1] == e.s1) return &e;
  }
  return nullptr;
}

// generated by build.py: launchers of the tensor-core multi-pass plans
#define CVB_GEMM(r0)                                               \
  int launch_gdA_##r0(const gd::Params&, int, cudaStream_t);       \
  int launch_gdB1_##r0(const gd::Params&, int, cudaStream_t);      \
  int launch_gdB2_##r0(const gd::Params&, int, cudaStream_t);      \
  int launch_gdC_##r0(const gd::Params&, int, cudaStream_t);
#include "gemm_registry.inc"
#undef CVB_GEMM
static const GdEntry kGemm[] = {
#define CVB_GEMM(r0) {r0, launch_gdA_##r0, launch_gdB1_##r0, launch_gdB2_##r0, launch_gdC_##r0},
#include "gemm_registry.inc"
#undef CVB_GEMM
};
static const GdEntry* find_gemm(const Plan1D& pl) {
  if (!pl.gemm) return nullptr;
  for (const GdEntry& e : kGemm)
    if (e.r0 == pl.radix[0]) return &e;
  return nullptr;
}

template <typename IO>
__global__ void __launch_bounds__(256) gd_epilogue_kernel(const gd::Params P) {
  gd::epilogue_body<IO>(P);
}

constexpr int kStripThreads = 256;

template <typename IO>
__global__ void __launch_bounds__(kStripThreads, 2) strip_colfwd_kernel(const StripParams SP) {
  extern __shared__ float2 smem[];
  strip_colfwd_body<IO>(SP, blockIdx.y, blockIdx.x, smem, 0);
}
__global__ void __launch_bounds__(kStripThreads, 2) strip_rowmid_kernel(const StripParams SP) {
  extern __shared__ float2 smem[];
  strip_rowmid_body(SP, blockIdx.y, blockIdx.x, smem, 0);
}
template <typename IO>
__global__ void __launch_bounds__(kStripThreads, 2) strip_colinv_kernel(const StripParams SP) {
  extern __shared__ float2 smem[];
  strip_colinv_body<IO>(SP, blockIdx.y, blockIdx.x, smem, 0);
}

namespace {
template <typename IO>
int launch_t(const FwdParams& P, void* workspace, size_t ws_bytes, cudaStream_t st,
             size_t ws_cap = kWorkspaceTarget, bool at_least_one = true) {
  const int npairs = num_pairs(P);
  // CVB_WS_MB: smaller chunks than the workspace allows (tuning aid; the caller's buffer is sized
  // for the default)
  const int ws_mb = CVB_TUNE("CVB_WS_MB", 0);
  if (ws_mb > 0 && ((size_t)ws_mb << 20) < ws_cap) ws_cap = (size_t)ws_mb << 20;
  const StripGeo g = strip_geometry(P.h, P.w, P.k, P.s, npairs, ws_cap, at_least_one);
  if (g.chunk_pairs < 1) return CVB_ERR_TOO_LARGE;
  if (!workspace || ws_bytes < g.ws_bytes) return CVB_ERR_WORKSPACE;
  if (P.py.gemm || P.px.gemm) {
    // tensor-core multi-pass kernels: four launches per chunk of pairs (and the epilogue at scale >= 2)
    const GdEntry* gy = find_gemm(P.py);
    const GdEntry* gx = find_gemm(P.px);
    if (!gy || !gx) return CVB_ERR_UNSUPPORTED_SIZE;
    const int io = sizeof(IO) == 4 ? CVB_F32 : CVB_BF16;
    gd::Params GP;
    GP.f = P;
    GP.ws = (float2*)workspace;
    GP.bmat = nullptr;
    // Pairs per launch: the cap keeps the chunk's workspace in L2; below it, the size whose tiles
    // (32 lines each, one resident block per tile slot) fill whole waves of the persistent blocks.
    int chunk = g.chunk_pairs;
    {
      const long long slots = (long long)sm_count() * ((P.py.radix[0] > 96 || P.px.radix[0] > 96) ? 1 : 2);
      double best = -1.0;
      for (int c2 = g.chunk_pairs; c2 >= (g.chunk_pairs + 1) / 2 && c2 >= 1; --c2) {
        long long work = 0, paid = 0;
        for (int p0 = 0; p0 < npairs; p0 += c2) {
          const long long np = (npairs - p0) < c2 ? (npairs - p0) : c2;
          for (int axis = 0; axis < 2; ++axis) {
            const long long tiles = (np * (axis ? P.h : P.w) + gd::kLines - 1) / gd::kLines;
            work += tiles;
            paid += ((tiles + slots - 1) / slots) * slots;
          }
        }
        const double eff = (double)work / (double)paid;
        if (eff > best + 1e-9) { best = eff; chunk = c2; }
      }
    }
    {
      const int forced = CVB_TUNE("CVB_GD_CHUNK", 0);
      if (forced > 0 && forced <= g.chunk_pairs) chunk = forced;
    }
    for (int p0 = 0; p0 < npairs; p0 += chunk) {
      GP.pair0 = p0;
      GP.npair = (npairs - p0) < chunk ? (npairs - p0) : chunk;
      int rc = gy->A(GP, io, st);
      if (rc == CVB_OK) rc = gx->B1(GP, io, st);
      if (rc == CVB_OK) rc = gx->B2(GP, io, st);
      if (rc == CVB_OK) rc = gy->C(GP, io, st);
      if (rc != CVB_OK) return rc;
      if (P.s > 1) {
        const long long cells = (long long)GP.npair * P.H * P.W;
        const int blocks = (int)std::min<long long>((cells + 255) / 256, (long long)sm_count() * 16);
        gd_epilogue_kernel<IO><<<blocks, 256, 0, st>>>(GP);
        CVB_CUDA(cudaGetLastError());
      }
    }
    return CVB_OK;
  }
  if (g.smem_col > kSmemLimit || g.smem_row > kSmemLimit) return CVB_ERR_UNSUPPORTED_SIZE;
  if (const int rc = allow_smem(strip_colfwd_kernel<IO>, g.smem_col)) return rc;
  if (const int rc = allow_smem(strip_colinv_kernel<IO>, g.smem_col)) return rc;
  if (const int rc = allow_smem(strip_rowmid_kernel, g.smem_row)) return rc;
  StripParams SP;
  SP.f = P;
  SP.ws = (float2*)workspace;
  SP.cw = g.cw; SP.rh = g.rh; SP.halo_l = g.halo_l; SP.halo_r = g.halo_r;
  SP.big_y = plan_has_big(P.py) ? 1 : 0;
  SP.big_x = plan_has_big(P.px) ? 1 : 0;
  rader_both(P.py, P.px, SP.ry, SP.rx);
  if (CVB_TUNE("CVB_NO_RADER", 0)) { SP.ry.R = 0; SP.rx.R = 0; }
  const int ncs = (P.w + g.cw - 1) / g.cw, nrs = (P.h + g.rh - 1) / g.rh;
  // compile-time axis plans when both axes have one (and the halo leaves room in a strip)
  const Strip2Entry* ey = find_strip2(P.py, SP.ry);
  const Strip2Entry* ex = find_strip2(P.px, SP.rx);
  const bool fast = ey && ex && g.halo_l + g.halo_r <= 4 && !CVB_TUNE("CVB_NO_STRIP2", 0);
  const int io_dtype = sizeof(IO) == 4 ? CVB_F32 : CVB_BF16;
  int chunk = g.chunk_pairs;
  if (fast && !CVB_TUNE("CVB_NO_BALANCE", 0)) {
    const int ly = strip2_lines(P.h, P.py.radix[0]), lx = strip2_lines(P.w, P.px.radix[0]);
    const int lc = ly - g.halo_l - g.halo_r;
    int ry[3] = {2, 2, 2}, rx[3] = {2, 2, 2};  // resident blocks per SM of A, B, C for each axis plan
    ey->Q(io_dtype, P.k, ry);
    ex->Q(io_dtype, P.k, rx);
    const int strips[3] = {(P.w + ly - 1) / ly, (P.h + lx - 1) / lx, (P.w + lc - 1) / lc};
    const int resident[3] = {ry[0], rx[1], ry[2]};
    chunk = balance_chunk(npairs, g.chunk_pairs, strips, resident, sm_count());
  }
  for (int p0 = 0; p0 < npairs; p0 += chunk) {
    SP.pair0 = p0;
    SP.npair = (npairs - p0) < chunk ? (npairs - p0) : chunk;
    if (fast) {
      int rc = ey->A(SP, io_dtype, st);
      if (rc == CVB_OK) rc = ex->B(SP, io_dtype, st);
      if (rc == CVB_OK) rc = ey->C(SP, io_dtype, st);
      if (rc != CVB_OK) return rc;
      continue;
    }
    strip_colfwd_kernel<IO><<<dim3(ncs, SP.npair), kStripThreads, g.smem_col, st>>>(SP);
    strip_rowmid_kernel<<<dim3(nrs, SP.npair), kStripThreads, g.smem_row, st>>>(SP);
    strip_colinv_kernel<IO><<<dim3(ncs, SP.npair), kStripThreads, g.smem_col, st>>>(SP);
    CVB_CUDA(cudaGetLastError());
  }
  return CVB_OK;
}
}  // namespace

// ---- scratch that nobody has to allocate -------------------------------------------
// Some callers of this library cannot call cudaMalloc (or any allocator) at the point
// where they run the operator: code inside a stream-ordered region whose memory pool is
// frozen, a plug-in that was handed only its input and output buffers, a latency-critical
// loop that must not touch the allocator lock.  For them the workspace of the multi-pass
// path lives here, in the library image: every GPU that loads the library holds these
// CVB_STATIC_SCRATCH_BYTES until the process exits.
//
// In host code `g_static_scratch` is only a handle for the runtime, not a device
// address; the address a kernel may use comes from cudaGetSymbolAddress, asked once per
// device with that device current.
static __device__ __align__(256) unsigned char g_static_scratch[CVB_STATIC_SCRATCH_BYTES];

int static_scratch_address(void** out) {
  static void* ptrs[64] = {nullptr};
  int dev = 0;
  CVB_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return CVB_ERR_BAD_ARGUMENT;
  if (!ptrs[dev]) {
    void* p = nullptr;
    CVB_CUDA(cudaGetSymbolAddress(&p, g_static_scratch));
    ptrs[dev] = p;
  }
  *out = ptrs[dev];
  return CVB_OK;
}

int launch_strip_static_scratch(const FwdParams& P, int io_dtype, cudaStream_t st) {
  void* scratch = nullptr;
  const int rc = static_scratch_address(&scratch);
  if (rc != CVB_OK) return rc;
  // the chunk of plane pairs is sized to the fixed array; a plane pair that does not fit is refused
  return io_dtype == CVB_F32
             ? launch_t<float>(P, scratch, CVB_STATIC_SCRATCH_BYTES, st, CVB_STATIC_SCRATCH_BYTES, false)
             : launch_t<__nv_bfloat16>(P, scratch, CVB_STATIC_SCRATCH_BYTES, st, CVB_STATIC_SCRATCH_BYTES, false);
}

int launch_strip(const FwdParams& P, int io_dtype, void* workspace, size_t ws_bytes, cudaStream_t st) {
  return io_dtype == CVB_F32 ? launch_t<float>(P, workspace, ws_bytes, st)
                             : launch_t<__nv_bfloat16>(P, workspace, ws_bytes, st);
}

}  // namespace cvb
