// Gradients of the real-plane solve (cvb_rp_bwd.cuh): kernels and launches.
#include "../../include/converse_b200.h"
#include "cvb_internal.h"
#include "cvb_rp_plan.h"
#include "cvb_rp_bwd.cuh"

namespace cvb {
namespace rp {

__global__ void __launch_bounds__(128, 4) rows_bwd_kernel(const __grid_constant__ BwdParams Q) {
  extern __shared__ float2 smem[];
  rows_bwd_body<kAnyRadix, 0>(Q, smem);
}
template <int K, int S>
__global__ void __launch_bounds__(256, AdjointTile<K, S>::blocks) adjoint_epilogue_kernel(const AdjointParams A) {
  extern __shared__ float4 tiles[];
  adjoint_epilogue_body<K, S>(A, (float*)tiles);
}
template <int K, int S>
static int launch_adjoint(AdjointParams A, int planes, cudaStream_t st) {
  plan_adjoint<K, S>(A);
  const size_t smem = (size_t)AdjointTile<K, S>::floats(A) * sizeof(float);
  if (const int rc = allow_smem(adjoint_epilogue_kernel<K, S>, smem)) return rc;
  adjoint_epilogue_kernel<K, S><<<planes, AdjointTile<K, S>::threads, smem, st>>>(A);
  return CVB_OK;
}
__global__ void __launch_bounds__(256) adjoint_epilogue_any_kernel(const AdjointParams A) {
  __shared__ float red[8];
  adjoint_epilogue_any(A, red);
}
__global__ void __launch_bounds__(256) pad_adjoint_kernel(const PadAdjointParams A) { pad_adjoint_body(A); }

// ------------------------------------------------------------------ chain rule from D to the taps and lambda
struct ChainParams {
  const float* weight;   // (C,k,k)
  const float* bias;     // (C)
  const float2* D;       // [nseg][C][w][hh]
  double* part;          // [row tiles][C][k k + 1]
  int C, k, s, h, w, hh, nseg;
  float eps;
};
constexpr int kChainRows = 32, kChainWarps = 8;
constexpr int kChainMaxScale = 4;

__device__ __forceinline__ double2 zmul(double2 a, double2 b) { return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ double2 zcis(long long m, int N) {   // exp(-2 pi i m / N)
  m %= N;
  if (m < 0) m += N;
  double2 r;
  sincospi(-2.0 * (double)m / (double)N, &r.y, &r.x);
  return r;
}
inline size_t chain_smem(int k, int s, int w) {
  return ((size_t)s * w * (k + 3) + (size_t)s * kChainRows * (k + 1)) * sizeof(double2) + (size_t)kChainWarps * (k * k + 1) * sizeof(double);
}

// One block: 32 rows k of one channel (a lane each), the frequencies f dealt to eight warps.  Per frequency the s x s
// aliases F of the kernel spectrum come from the separable exponentials; with d = fold |F|^2 + lambda and D the cross
// spectrum, dL = Re sum_alias A dF with
//   s = 1:  A = conj(D) / d - 2 Re(D (conj F + lambda)) / d^2 conj F           (M = (conj F + lambda) / d)
//   s > 1:  A = -(D box + 2 Re(D M) conj F) / (s^2 d)                           (M = (1 - fold(F box)) / d)
// and dF = sum_ab dK[a][b] ey^(a-c) ex^(b-c): every lane sums A ex^(b-c) over its frequencies, then the taps of its row.
// fp64; the rows k = 0 and k = h / 2 stand for themselves, the others for their mirror rows too.
template <int CK, int CS>
__global__ void __launch_bounds__(256) chain_kernel(const ChainParams T) {
  extern __shared__ double2 csm[];
  constexpr int AS = CS ? CS : kChainMaxScale, AK = CK ? CK : kMaxTaps;
  const int s = CS ? CS : T.s, k = CK ? CK : T.k, w = T.w, cc = k / 2, Nh = s * T.h, Nw = s * w;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, c = blockIdx.y, k0 = blockIdx.x * kChainRows;
  double2* tx = csm;                          // [ib][f][a]
  double2* e0 = tx + (size_t)s * w * k;       // [ib][f]: ex^-c
  double2* e1 = e0 + s * w;                   // [ib][f]: ex
  double2* dw = e1 + s * w;                   // [ib][f]: box
  double2* ey = dw + s * w;                   // [ia][row][a]
  double2* dh = ey + s * kChainRows * k;      // [ia][row]
  double* red = (double*)(dh + s * kChainRows);
  const float* K = T.weight + (size_t)c * k * k;
  for (int i = tid; i < s * w; i += 256) {
    const int V = i;                          // f + ib w
    const double2 e = zcis(V, Nw), p0 = zcis(-(long long)cc * V, Nw);
    e0[i] = p0; e1[i] = e;
    double2 d = make_double2(0.0, 0.0), q = make_double2(1.0, 0.0);
    for (int b = 0; b < s; ++b) { d.x += q.x; d.y += q.y; q = zmul(q, e); }
    dw[i] = d;
    for (int a = 0; a < k; ++a) {
      double2 p = p0, sum = make_double2(0.0, 0.0);
      for (int b = 0; b < k; ++b) {
        const double kv = (double)K[a * k + b];
        sum.x += kv * p.x; sum.y += kv * p.y;
        p = zmul(p, e);
      }
      tx[(size_t)i * k + a] = sum;
    }
  }
  for (int i = tid; i < s * kChainRows; i += 256) {
    const int row = i % kChainRows, ia = i / kChainRows, U = k0 + row + ia * T.h;
    const double2 e = zcis(U, Nh);
    double2 p = zcis(-(long long)cc * U, Nh), d = make_double2(0.0, 0.0), q = make_double2(1.0, 0.0);
    for (int a = 0; a < k; ++a) { ey[i * k + a] = p; p = zmul(p, e); }
    for (int a = 0; a < s; ++a) { d.x += q.x; d.y += q.y; q = zmul(q, e); }
    dh[i] = d;
  }
  __syncthreads();
  const double lam = 1.0 / (1.0 + exp(-((double)T.bias[c] - 9.0))) + (double)T.eps;
  const int row = k0 + lane;
  const double wgt = row >= T.hh ? 0.0 : (row == 0 || 2 * row == T.h) ? 1.0 : 2.0;
  const int krow = row < T.hh ? row : T.hh - 1;
  const double is2 = 1.0 / (double)(s * s);
  double2 S[AS][AK];
  double glam = 0.0;
#pragma unroll
  for (int ia = 0; ia < AS; ++ia)
#pragma unroll
    for (int b = 0; b < AK; ++b) S[ia][b] = make_double2(0.0, 0.0);
  for (int f = warp; f < w; f += kChainWarps) {
    double2 D = make_double2(0.0, 0.0);
    for (int sg = 0; sg < T.nseg; ++sg) {
      const float2 v = __ldg(T.D + ((size_t)(sg * T.C + c) * w + f) * T.hh + krow);
      D.x += v.x; D.y += v.y;
    }
    double2 F[AS][AS];
    double nr = 0.0, ni = 0.0, den = 0.0;
#pragma unroll
    for (int ia = 0; ia < (CS ? CS : s); ++ia)
#pragma unroll
      for (int ib = 0; ib < (CS ? CS : s); ++ib) {
        const double2* pe = ey + (ia * kChainRows + lane) * k;
        const double2* pt = tx + (size_t)(ib * w + f) * k;
        double fr = 0.0, fi = 0.0;
#pragma unroll
        for (int a = 0; a < (CK ? CK : k); ++a) {
          fr += pe[a].x * pt[a].x - pe[a].y * pt[a].y;
          fi += pe[a].x * pt[a].y + pe[a].y * pt[a].x;
        }
        F[ia][ib] = make_double2(fr, fi);
        den += fr * fr + fi * fi;
        if (s > 1) {
          const double2 d = zmul(dh[ia * kChainRows + lane], dw[ib * w + f]);
          nr += fr * d.x - fi * d.y;
          ni += fr * d.y + fi * d.x;
        }
      }
    const double d = den * is2 + lam, inv = 1.0 / d;
    double2 M;
    if (s == 1) M = make_double2((F[0][0].x + lam) * inv, -F[0][0].y * inv);
    else M = make_double2((1.0 - nr * is2) * inv, -ni * is2 * inv);
    const double t = D.x * M.x - D.y * M.y;       // Re(D M)
    if (s == 1) glam += (D.x - t) * inv;          // d/dlambda: Re(D (1 - M)) / d
    else glam -= t * inv;
#pragma unroll
    for (int ia = 0; ia < (CS ? CS : s); ++ia)
#pragma unroll
      for (int ib = 0; ib < (CS ? CS : s); ++ib) {
        const double2 Fv = F[ia][ib];
        double2 A;
        if (s == 1) {
          A = make_double2((D.x - 2.0 * t * Fv.x) * inv, (-D.y + 2.0 * t * Fv.y) * inv);
        } else {
          const double2 box = zmul(dh[ia * kChainRows + lane], dw[ib * w + f]);
          const double2 db = zmul(D, box);
          A = make_double2(-(db.x + 2.0 * t * Fv.x) * is2 * inv, -(db.y - 2.0 * t * Fv.y) * is2 * inv);
        }
        double2 q = zmul(A, e0[ib * w + f]);
        const double2 e = e1[ib * w + f];
#pragma unroll
        for (int b = 0; b < (CK ? CK : k); ++b) {
          S[ia][b].x += q.x; S[ia][b].y += q.y;
          q = zmul(q, e);
        }
      }
  }
  const int nt = k * k + 1;
  auto warp_sum = [&](double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  };
#pragma unroll
  for (int a = 0; a < (CK ? CK : k); ++a)
#pragma unroll
    for (int b = 0; b < (CK ? CK : k); ++b) {
      double v = 0.0;
#pragma unroll
      for (int ia = 0; ia < (CS ? CS : s); ++ia) {
        const double2 p = ey[(ia * kChainRows + lane) * k + a];
        v += p.x * S[ia][b].x - p.y * S[ia][b].y;
      }
      v = warp_sum(v * wgt);
      if (lane == 0) red[warp * nt + a * k + b] = v;
    }
  glam = warp_sum(glam * wgt);
  if (lane == 0) red[warp * nt + k * k] = glam;
  __syncthreads();
  for (int i = tid; i < nt; i += 256) {
    double v = 0.0;
    for (int j = 0; j < kChainWarps; ++j) v += red[j * nt + i];
    T.part[((size_t)blockIdx.x * T.C + c) * nt + i] = v;
  }
}

struct FinishParams {
  const double* part;
  const float* taps;     // [B C][k k] or null
  const float* bias;
  float* gw;             // (C,k,k)
  float* gb;             // (C)
  int tiles, B, C, k;
  double scale;          // 1 / (4 h w): D is four times the cross spectrum
};
__global__ void __launch_bounds__(128) finish_kernel(const FinishParams F) {
  const int c = blockIdx.x, kk = F.k * F.k;
  for (int i = threadIdx.x; i <= kk; i += 128) {
    double v = 0.0;
    for (int t = 0; t < F.tiles; ++t) v += F.part[((size_t)t * F.C + c) * (kk + 1) + i];
    v *= F.scale;
    if (i < kk) {
      if (F.taps)
        for (int b = 0; b < F.B; ++b) v += (double)F.taps[((size_t)b * F.C + c) * kk + i];
      F.gw[(size_t)c * kk + i] = (float)v;
    } else {
      const double sg = 1.0 / (1.0 + exp(-((double)F.bias[c] - 9.0)));
      F.gb[c] = (float)(v * sg * (1.0 - sg));
    }
  }
}

// rows_bwd_body with a matrix stage, by width (k_rp_matrix.cu)
typedef int (*BwdLauncher)(const BwdParams&, dim3, size_t, cudaStream_t);
#define CVB_RP_X(M) int launch_matrix_rows_bwd_##M(const BwdParams&, dim3, size_t, cudaStream_t);
CVB_RP_EACH_WIDTH(CVB_RP_X)
#undef CVB_RP_X
static BwdLauncher matrix_bwd(int width) {
  switch (width) {
#define CVB_RP_X(M) case M: return launch_matrix_rows_bwd_##M;
    CVB_RP_EACH_WIDTH(CVB_RP_X)
#undef CVB_RP_X
  }
  return nullptr;
}

static size_t rows_bwd_smem(const Params& P) {
  const size_t tile = ((size_t)P.pitch * kLines + 1) & ~(size_t)1;
  return 3 * tile * sizeof(float2) + (P.ax.mp ? matrix_entries(P.ax.r0) : 0) * sizeof(float);
}

// Device buffers of one backward call, carved out of one workspace
struct BwdPlan {
  size_t wx, wg, v, f, D, taps, part, total;
  int nseg, tiles;
};
static bool plan_bwd(const Params& P, int sms, bool want_x, bool want_params, BwdPlan& b) {
  auto up = [](size_t n) { return (n + 255) / 256 * 256; };
  const size_t planes = (size_t)P.B * P.C, spec = up(planes * P.hh * P.wp * sizeof(float2));
  const bool direct = P.s == 1 && P.p == 0;          // the solved cotangent is dL/dx itself
  const int groups = ((P.hh + kLines - 1) / kLines) * P.C;
  b.nseg = 1;
  while (b.nseg < P.B && groups * b.nseg < 3 * sms) ++b.nseg;
  b.tiles = (P.hh + kChainRows - 1) / kChainRows;
  size_t at = 0;
  auto take = [&](size_t n) { const size_t o = at; at += up(n); return o; };
  b.wx = take(want_params ? spec : 0);
  b.wg = take(spec);
  b.v = take(P.s > 1 ? planes * P.h * P.w * sizeof(float) : 0);
  b.f = take(want_x && !direct ? planes * P.h * P.w * sizeof(float) : 0);
  b.D = take(want_params ? (size_t)b.nseg * P.C * P.w * P.hh * sizeof(float2) : 0);
  b.taps = take(want_params && P.s > 1 ? planes * P.k * P.k * sizeof(float) : 0);
  b.part = take(want_params ? (size_t)b.tiles * P.C * (P.k * P.k + 1) * sizeof(double) : 0);
  b.total = at;
  if (planes > 0x7fffffff / P.wc || planes > 0x7fffffff / P.hh) return false;
  if (cols_smem(P) > kSmemLimit || rows_smem(P) > kSmemLimit) return false;
  if (!want_params) return true;
  return rows_bwd_smem(P) <= kSmemLimit && P.s <= kChainMaxScale && chain_smem(P.k, P.s, P.w) <= kSmemLimit && P.C <= 65535;
}

size_t bwd_workspace(int B, int C, int H, int W, int k, int s, int p, bool want_x, bool want_params, int sms) {
  Params P;
  BwdPlan b;
  if (!fill_params(P, nullptr, B, C, H, W, k, s, p, 0) || !plan_bwd(P, sms, want_x, want_params, b)) return 0;
  return b.total;
}

// Tap counts and scales of chain_kernel with its sums in registers: those that networks train at.  At scales 3 and 4 the s k
// double-precision sums would not fit (7 x 3: 84 registers for the sums alone, beside the 36 of the aliases), so the
// run-time form, whose sums are in local memory, serves them: a training step of 8 x 64 planes of 32 x 32 takes 195 us at
// scale 3 or 4 with 3 x 3 taps and 167 us at scale 2 with 5 x 5; 351 us with 7 x 7 taps at scale 4.
#define CVB_CHAIN_CASES(X) X(3, 1) X(5, 1) X(7, 1) X(2, 2) X(3, 2) X(5, 2) X(7, 2)

int run_bwd(const float* x, const float* g, const float* r, const void* table, const float* weight, const float* bias,
            float* gx, float* gw, float* gb, int B, int C, int H, int W, int k, int s, int p, int pad_mode, float eps,
            void* workspace, size_t ws_bytes, int sms, cudaStream_t st) {
  const bool want_x = gx != nullptr, want_params = gw != nullptr;
  Params P;
  BwdPlan b;
  if (!fill_params(P, table, B, C, H, W, k, s, p, pad_mode) || !plan_bwd(P, sms, want_x, want_params, b))
    return CVB_ERR_UNSUPPORTED_SIZE;
  if (!workspace || ws_bytes < b.total) return CVB_ERR_WORKSPACE;
  char* base = (char*)workspace;
  const int planes = B * C;
  int rc = CVB_OK;
  // row spectra of y
  if (want_params) {
    Params Y = P;
    Y.s = 1;
    Y.x = x;
    Y.ws = (float2*)(base + b.wx);
    rc = cols_fwd(Y, planes, st);
    if (rc != CVB_OK) return rc;
  }
  // q and its column spectra
  Params Q = P;
  Q.s = 1;
  Q.ws = (float2*)(base + b.wg);
  Q.conj = 1;
  if (s == 1) {
    Q.x = g;
    Q.pad_mode = CVB_PAD_CONSTANT;     // the cotangent extended by zeros
  } else {
    AdjointParams A;
    A.g = g; A.r = want_params ? r : nullptr; A.weight = weight;
    A.v = (float*)(base + b.v); A.taps = want_params ? (float*)(base + b.taps) : nullptr;
    A.C = C; A.H = H; A.W = W; A.k = k; A.s = s; A.p = p; A.h = P.h; A.w = P.w; A.wp = P.wp;
    if (want_params && !r) return CVB_ERR_BAD_ARGUMENT;
    // the tap counts of the networks (2 at scale 2, 3, 5, 7) at the scales that have parameter gradients; others read g once
    // per tap
    switch (s * 16 + k) {
#define X(KK, SS) case SS * 16 + KK: rc = launch_adjoint<KK, SS>(A, planes, st); break;
      X(2, 2) X(3, 2) X(5, 2) X(7, 2) X(3, 3) X(5, 3) X(7, 3) X(3, 4) X(5, 4) X(7, 4)
#undef X
      default: adjoint_epilogue_any_kernel<<<planes, 256, 0, st>>>(A);
    }
    if (rc != CVB_OK) return rc;
    CVB_CUDA(cudaGetLastError());
    Q.x = A.v;
    Q.H = P.h; Q.W = P.w; Q.p = 0;
    Q.pad_mode = CVB_PAD_CIRCULAR;
  }
  rc = cols_fwd(Q, planes, st);
  if (rc != CVB_OK) return rc;
  // along x: cross spectrum, and the cotangent through the conjugated multiplier
  if (want_params) {
    BwdParams R;
    R.P = Q;
    R.wx = (const float2*)(base + b.wx);
    R.D = (float2*)(base + b.D);
    R.nseg = b.nseg;
    R.solve = want_x ? 1 : 0;
    const dim3 grid((P.hh + kLines - 1) / kLines, C, b.nseg);
    const size_t smem = rows_bwd_smem(P);
    if (P.ax.mp) {
      rc = matrix_bwd(P.ax.mp)(R, grid, smem, st);
      if (rc != CVB_OK) return rc;
    } else {
      rc = allow_smem(rows_bwd_kernel, smem);
      if (rc != CVB_OK) return rc;
      rows_bwd_kernel<<<grid, 128, smem, st>>>(R);
      CVB_CUDA(cudaGetLastError());
    }
  } else {
    rc = rows(Q, planes, st);
    if (rc != CVB_OK) return rc;
  }
  if (want_x) {
    const bool direct = s == 1 && p == 0;
    Params O = Q;
    O.po = 0; O.OH = P.h; O.OW = P.w;
    O.out = direct ? gx : (float*)(base + b.f);
    rc = cols_inv(O, planes, st);
    if (rc != CVB_OK) return rc;
    if (!direct) {
      PadAdjointParams A;
      A.f = (const float*)O.out; A.g = s > 1 ? g : nullptr; A.gx = gx;
      A.H = H; A.W = W; A.s = s; A.p = p; A.h = P.h; A.w = P.w; A.pad_mode = pad_mode;
      for (int p0 = 0; p0 < planes; p0 += 65535) {
        const int np = planes - p0 < 65535 ? planes - p0 : 65535;
        PadAdjointParams Z = A;
        Z.f += (size_t)p0 * P.h * P.w; Z.gx += (size_t)p0 * H * W;
        if (Z.g) Z.g += (size_t)p0 * s * s * H * W;
        pad_adjoint_kernel<<<dim3((H * W + 1023) / 1024, np), 256, 0, st>>>(Z);
      }
      CVB_CUDA(cudaGetLastError());
    }
  }
  if (want_params) {
    ChainParams T;
    T.weight = weight; T.bias = bias; T.D = (const float2*)(base + b.D); T.part = (double*)(base + b.part);
    T.C = C; T.k = k; T.s = s; T.h = P.h; T.w = P.w; T.hh = P.hh; T.nseg = b.nseg; T.eps = eps;
    const size_t smem = chain_smem(k, s, P.w);
    const dim3 grid(b.tiles, C);
    switch (s * 16 + k) {
#define X(KK, SS)                                                                                                  \
      case SS * 16 + KK:                                                                                           \
        rc = allow_smem(chain_kernel<KK, SS>, smem);                                                               \
        if (rc != CVB_OK) return rc;                                                                               \
        chain_kernel<KK, SS><<<grid, 256, smem, st>>>(T);                                                          \
        break;
      CVB_CHAIN_CASES(X)
#undef X
      default:
        rc = allow_smem(chain_kernel<0, 0>, smem);
        if (rc != CVB_OK) return rc;
        chain_kernel<0, 0><<<grid, 256, smem, st>>>(T);
    }
    CVB_CUDA(cudaGetLastError());
    FinishParams F;
    F.part = T.part; F.taps = s > 1 ? (const float*)(base + b.taps) : nullptr; F.bias = bias; F.gw = gw; F.gb = gb;
    F.tiles = b.tiles; F.B = B; F.C = C; F.k = k; F.scale = 0.25 / ((double)P.h * (double)P.w);
    finish_kernel<<<C, 128, 0, st>>>(F);
    CVB_CUDA(cudaGetLastError());
  }
  return CVB_OK;
}

}  // namespace rp
}  // namespace cvb
