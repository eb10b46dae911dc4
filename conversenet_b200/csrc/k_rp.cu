// Real-plane solve (cvb_rp.cuh): table build and launches.
#include "../../include/converse_b200.h"
#include "cvb_internal.h"
#include "cvb_rp_plan.h"

namespace cvb {
namespace rp {

// generated launchers: register plans (k_rp_cols.cu, k_rp_rows.cu), matrix stages by width (k_rp_matrix.cu)
int launch_cols_fwd_f32(const Params&, bool, int, int, size_t, cudaStream_t);
int launch_cols_fwd_bf16(const Params&, bool, int, int, size_t, cudaStream_t);
int launch_cols_inv_f32(const Params&, bool, int, int, size_t, cudaStream_t);
int launch_cols_inv_bf16(const Params&, bool, int, int, size_t, cudaStream_t);
int launch_epilogue_f32(const Params&, cudaStream_t);
int launch_epilogue_bf16(const Params&, cudaStream_t);
int launch_rows(const Params&, bool, int, int, size_t, cudaStream_t);
int launch_plane_f32(const Params&, bool, int, size_t, cudaStream_t);
int launch_plane_bf16(const Params&, bool, int, size_t, cudaStream_t);
int launch_fix(int kind, const Params&, int io_dtype, int sms, cudaStream_t);   // integer contractions (k_fix.cu)
typedef int (*MatrixLauncher)(const Params&, int, int, int, size_t, cudaStream_t);   // (.., tensor type, threads, grid, ..)
struct MatrixEntry { int width; MatrixLauncher cols_fwd, rows, cols_inv; };
#define CVB_RP_X(M)                                                            \
  int launch_matrix_cols_fwd_##M(const Params&, int, int, int, size_t, cudaStream_t); \
  int launch_matrix_rows_##M(const Params&, int, int, int, size_t, cudaStream_t);     \
  int launch_matrix_cols_inv_##M(const Params&, int, int, int, size_t, cudaStream_t);
CVB_RP_EACH_WIDTH(CVB_RP_X)
#undef CVB_RP_X
static const MatrixEntry kMatrix[] = {
#define CVB_RP_X(M) {M, launch_matrix_cols_fwd_##M, launch_matrix_rows_##M, launch_matrix_cols_inv_##M},
  CVB_RP_EACH_WIDTH(CVB_RP_X)
#undef CVB_RP_X
};
static const MatrixEntry& matrix_entry(int width) {
  int i = 0;
  while (kMatrix[i].width != width) ++i;
  return kMatrix[i];
}

// ------------------------------------------------------------------ table
struct TableParams {
  const float* weight;   // (C,k,k)
  const float* bias;     // (C)
  float2* out;
  int C, k, s, h, w, hh, kind;
  float eps;
  int tk, tf;            // tiles of 32 rows, of 16 frequencies along x
  int r0y, r1y, r0x, r1x, ey, ex;  // plans; entries of the matrix stages (0 = none)
  size_t tw, twy, twx, dmy, dmx, fixy, fixx;
  int fy, fx;                      // values of the operands of the integer contractions (0 = none)
};
constexpr int kTK = 32, kTF = 16;

__device__ __forceinline__ double2 cmul(double2 a, double2 b) { return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
// exp(-2 pi i m / N)
__device__ __forceinline__ double2 cis(long long m, int N) {
  m %= N;
  if (m < 0) m += N;
  double2 r;
  sincospi(-2.0 * (double)m / (double)N, &r.y, &r.x);
  return r;
}

// Operand of the integer contractions along an axis of length N: value i = (parity, cosine / sine, row, q < 64), three
// digits; then the fp32 values q = 64 .. 67 of every row.
__device__ void fix_value_out(unsigned char* out, int N, int i) {
  const int nr = fix_rows(N), M = N / 2, QH = M / 2;
  const bool whole = i >= 256 * nr;
  const int e = whole ? i - 256 * nr : i, per = whole ? 4 : 64;
  const int q = e % per + (whole ? 64 : 0), j = (e / per) % nr, cs = (e / (per * nr)) & 1, par = e / (2 * per * nr), k = 2 * j + par;
  double sn, cn;
  sincospi(2.0 * (double)((q * k) % N) / (double)N, &sn, &cn);
  double v = k <= M && q <= QH ? (cs ? sn : cn) : 0.0;
  if (q == 0 || 2 * q == M) v *= 0.5;
  if (whole) {
    ((float*)(out + fix_operand(N)))[((par * 2 + cs) * 4 + q - 64) * nr + j] = (float)v;
    return;
  }
  const int n = __double2int_rn(v / (double)kFixUnit);
  const uint32_t t = ((uint32_t)n + 0x808080u) ^ 0x808080u;
  int step;
  const int o = fix_row_offset(nr, par, cs, j, q, step);
  out[o] = (unsigned char)(t >> 16); out[o + step] = (unsigned char)(t >> 8); out[o + 2 * step] = (unsigned char)t;
}

// twiddles, matrix rows and contraction operands behind the multiplier
__device__ void table_tail(const TableParams& T, int i0, int step) {
  const int nt = T.h + T.w;
  for (int i = i0; i < T.fy + T.fx; i += step) {
    if (i < T.fy) fix_value_out((unsigned char*)(T.out + T.fixy), T.h, i);
    else fix_value_out((unsigned char*)(T.out + T.fixx), T.w, i - T.fy);
  }
  for (int i = i0; i < 2 * nt + T.ey + T.ex; i += step) {
    double sn, cs;
    if (i < 2 * nt) {
      const int t = i < nt ? i : i - nt, N = t < T.h ? T.h : T.w, n = t < T.h ? t : t - T.h;
      const int r1 = t < T.h ? T.r1y : T.r1x, m = i < nt ? n : (n / r1) * (n % r1);   // position k0 r1 + j: k0 j
      sincospi(2.0 * (double)m / (double)N, &sn, &cs);
      T.out[(i < nt ? T.tw + (t < T.h ? 0 : T.h) : t < T.h ? T.twy : T.twx) + n] = make_float2((float)cs, (float)sn);
    } else {
      const bool y = i < 2 * nt + T.ey;
      const int e = y ? i - 2 * nt : i - 2 * nt - T.ey, R = y ? T.r0y : T.r0x;
      const int mp = matrix_width(R), n = (R / 2 + 1) * mp, sine = e >= n, f = sine ? e - n : e;
      const int k = f / mp, q = f % mp + 1;
      sincospi(2.0 * (double)((q * k) % R) / (double)R, &sn, &cs);
      ((float*)(T.out + (y ? T.dmy : T.dmx)))[e] = q > R / 2 ? 0.f : (float)(sine ? sn : cs);
    }
  }
}

// Multiplier rows k = 0 .. h/2, [c][f][k], fp64, times 1 / (2 h w): the separated column spectra are twice the
// transforms.  A block computes 32 rows x 16 frequencies of one channel from the separable exponentials
//   FK[U,V] = sum_a ey^(a-c) ( sum_b K[a][b] ex^(b-c) ),  U = k + ia h, V = f + ib w,
// whose two halves are computed once per block into shared memory.
__global__ void __launch_bounds__(256) table_kernel(const TableParams T) {
  extern __shared__ double2 tsm[];
  const int tid = threadIdx.x, nb = T.C * T.tk * T.tf;
  if (blockIdx.x >= nb) {
    table_tail(T, (blockIdx.x - nb) * 256 + tid, (gridDim.x - nb) * 256);
    return;
  }
  const int s = T.s, k = T.k, cc = k / 2, Nh = s * T.h, Nw = s * T.w;
  const int c = blockIdx.x / (T.tk * T.tf), rest = blockIdx.x % (T.tk * T.tf);
  const int k0 = (rest % T.tk) * kTK, f0 = (rest / T.tk) * kTF;
  double2* tx = tsm;                       // [ib][f][a]
  double2* ey = tx + s * kTF * k;          // [ia][row][a]
  double2* dw = ey + s * kTK * k;          // [ib][f]
  double2* dh = dw + s * kTF;              // [ia][row]
  double2* lam = dh + s * kTK;
  const float* K = T.weight + (size_t)c * k * k;
  if (tid == 0) lam->x = 1.0 / (1.0 + exp(-((double)T.bias[c] - 9.0))) + (double)T.eps;
  for (int i = tid; i < s * kTF * k; i += 256) {
    const int a = i % k, f = (i / k) % kTF, ib = i / (k * kTF);
    const int V = f0 + f + ib * T.w;
    const double2 e = cis(V, Nw);
    double2 p = cis(-(long long)cc * V, Nw), sum = make_double2(0.0, 0.0);
    for (int b = 0; b < k; ++b) {
      const double kv = (double)K[a * k + b];
      sum.x += kv * p.x; sum.y += kv * p.y;
      p = cmul(p, e);
    }
    tx[i] = sum;
    if (a == 0) {
      double2 d = make_double2(0.0, 0.0), q = make_double2(1.0, 0.0);
      for (int b = 0; b < s; ++b) { d.x += q.x; d.y += q.y; q = cmul(q, e); }
      dw[ib * kTF + f] = d;
    }
  }
  for (int i = tid; i < s * kTK; i += 256) {
    const int row = i % kTK, ia = i / kTK, U = k0 + row + ia * T.h;
    const double2 e = cis(U, Nh);
    double2 p = cis(-(long long)cc * U, Nh), d = make_double2(0.0, 0.0), q = make_double2(1.0, 0.0);
    for (int a = 0; a < k; ++a) { ey[i * k + a] = p; p = cmul(p, e); }
    for (int a = 0; a < s; ++a) { d.x += q.x; d.y += q.y; q = cmul(q, e); }
    dh[i] = d;
  }
  __syncthreads();
  const double norm = 0.5 / ((double)T.h * (double)T.w), ia2 = 1.0 / (double)(s * s);
  for (int e = tid; e < kTK * kTF; e += 256) {
    const int row = e % kTK, f = e / kTK;
    if (k0 + row >= T.hh || f0 + f >= T.w) continue;
    double nr = 0.0, ni = 0.0, den = 0.0;
    for (int ia = 0; ia < s; ++ia)
      for (int ib = 0; ib < s; ++ib) {
        const double2* pe = ey + (ia * kTK + row) * k;
        const double2* pt = tx + (ib * kTF + f) * k;
        double fr = 0.0, fi = 0.0;
        for (int a = 0; a < k; ++a) {
          fr += pe[a].x * pt[a].x - pe[a].y * pt[a].y;
          fi += pe[a].x * pt[a].y + pe[a].y * pt[a].x;
        }
        den += fr * fr + fi * fi;
        if (s == 1) {
          nr = fr; ni = -fi;
        } else {
          const double2 d = cmul(dh[ia * kTK + row], dw[ib * kTF + f]);
          nr += fr * d.x - fi * d.y;
          ni += fr * d.y + fi * d.x;
        }
      }
    const double d = den * ia2 + lam->x, inv = norm / d;
    double tr, ti;
    if (T.kind == 1) { tr = inv; ti = 0.0; }
    else if (s == 1) { tr = (nr + lam->x) * inv; ti = ni * inv; }
    else { tr = (1.0 - nr * ia2) * inv; ti = -ni * ia2 * inv; }
    T.out[((size_t)c * T.w + f0 + f) * T.hh + k0 + row] = make_float2((float)tr, (float)ti);
  }
}

// scales whose alias arrays do not fit the tiled kernel's shared memory: one thread per entry
__global__ void table_slow_kernel(const TransferParams S, const TableParams T) {
  const size_t total = (size_t)T.C * T.w * T.hh;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int k = (int)(i % T.hh);
    const size_t rest = i / T.hh;
    double tr, ti;
    transfer_value_slow(S, (int)(rest / T.w), k, (int)(rest % T.w), tr, ti);
    const double norm = 0.5 / ((double)T.h * (double)T.w);
    T.out[i] = make_float2((float)(tr * norm), (float)(ti * norm));
  }
  table_tail(T, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

size_t table_bytes(int C, int h, int w) {
  int r0y, r1y, r0x, r1x;
  if (!axis_plan(h, r0y, r1y) || !axis_plan(w, r0x, r1x)) return 0;
  return blob_layout(C, h, w, r0y, r0x).total * sizeof(float2);
}

int build_table(const float* weight, const float* bias, int C, int k, int s, int h, int w, float eps, int kind,
                void* table, cudaStream_t st) {
  int r0y, r1y, r0x, r1x;
  if (!axis_plan(h, r0y, r1y) || !axis_plan(w, r0x, r1x)) return CVB_ERR_UNSUPPORTED_SIZE;
  const Blob bl = blob_layout(C, h, w, r0y, r0x);
  TableParams T;
  T.weight = weight; T.bias = bias; T.out = (float2*)table;
  T.C = C; T.k = k; T.s = s; T.h = h; T.w = w; T.hh = h / 2 + 1; T.kind = kind; T.eps = eps;
  T.tk = (T.hh + kTK - 1) / kTK; T.tf = (w + kTF - 1) / kTF;
  T.r0y = r0y; T.r1y = r1y; T.r0x = r0x; T.r1x = r1x; T.ey = matrix_entries(r0y); T.ex = matrix_entries(r0x);
  T.tw = bl.tw; T.twy = bl.twy; T.twx = bl.twx; T.dmy = bl.dmy; T.dmx = bl.dmx; T.fixy = bl.fixy; T.fixx = bl.fixx;
  T.fy = fix_axis(h, r0y) ? 272 * fix_rows(h) : 0; T.fx = fix_axis(w, r0x) ? 272 * fix_rows(w) : 0;
  const int tail = (std::max(2 * (h + w) + T.ey + T.ex, T.fy + T.fx) + 255) / 256;
  const size_t smem = (size_t)(s * (kTF + kTK) * (k + 1) + 1) * sizeof(double2);
  const long long nblk = (long long)C * T.tk * T.tf;
  if (nblk + tail > 0x7fffffffLL) return CVB_ERR_TOO_LARGE;
  if (smem <= 48 * 1024) {
    table_kernel<<<(int)nblk + tail, 256, smem, st>>>(T);
  } else {
    TransferParams S;
    memset(&S, 0, sizeof(S));
    S.weight = weight; S.bias = bias; S.C = C; S.k = k; S.s = s; S.h = h; S.w = w; S.eps = eps; S.kind = kind;
    table_slow_kernel<<<148 * 16, 128, 0, st>>>(S, T);
  }
  CVB_CUDA(cudaGetLastError());
  return CVB_OK;
}

// ------------------------------------------------------------------ forward
static void set_vec(Params& P, bool f32) {
  P.vec = P.p % 2 == 0 && P.W % 2 == 0 && ((size_t)P.x) % (f32 ? 8 : 4) == 0;
  P.vec_out = P.po % 2 == 0 && P.OW % 2 == 0 && ((size_t)P.out) % (f32 ? 8 : 4) == 0;
}

// one launch of each strip kernel over planes 0 .. planes - 1 (fp32 tensors)
static int strip(Params& P, int planes, int which, cudaStream_t st) {
  set_vec(P, true);
  P.plane0 = 0; P.nplane = planes; P.status = status_ptr();
  if (takes_fix(P, which, sm_count())) return launch_fix(which, P, CVB_F32, sm_count(), st);
  const int gc = (planes * P.wc + kLines - 1) / kLines, gr = (planes * P.hh + kLines - 1) / kLines;
  const int tc = strip_threads(P, false, gc, sm_count()), tr = strip_threads(P, true, gr, sm_count());
  if (which == 1)
    return P.ax.mp ? matrix_entry(P.ax.mp).rows(P, CVB_F32, tr, gr, rows_smem(P), st)
                   : launch_rows(P, small_axis(P.ax), tr, gr, rows_smem(P), st);
  if (P.ay.mp)
    return (which == 0 ? matrix_entry(P.ay.mp).cols_fwd : matrix_entry(P.ay.mp).cols_inv)(P, CVB_F32, tc, gc, cols_smem(P), st);
  return (which == 0 ? launch_cols_fwd_f32 : launch_cols_inv_f32)(P, small_axis(P.ay), tc, gc, cols_smem(P), st);
}
int cols_fwd(Params& P, int planes, cudaStream_t st) { return strip(P, planes, 0, st); }
int rows(Params& P, int planes, cudaStream_t st) { return strip(P, planes, 1, st); }
int cols_inv(Params& P, int planes, cudaStream_t st) { return strip(P, planes, 2, st); }

int run(Params& P, const Route& r, int io_dtype, void* workspace, size_t ws_bytes, cudaStream_t st) {
  const bool f32 = io_dtype == CVB_F32;
  const int planes = P.B * P.C;
  set_vec(P, f32);
  if (r.one_block) {
    P.plane0 = 0; P.nplane = planes;
    const size_t smem = plane_smem(P.h, P.w, P.k);
    // planes that leave SMs idle take the wide block (up to 512 threads, 128 registers)
    const bool wide = planes <= sm_count();
    const bool small = !wide && small_axis(P.ay) && small_axis(P.ax);
    const int threads = plane_threads(P, wide ? 512 : 256, planes > 2 * sm_count());
    return f32 ? launch_plane_f32(P, small, threads, smem, st) : launch_plane_bf16(P, small, threads, smem, st);
  }
  if (r.chunk < 1) return CVB_ERR_TOO_LARGE;
  if (!workspace || ws_bytes < r.ws_bytes) return CVB_ERR_WORKSPACE;
  const size_t smem_c = cols_smem(P), smem_r = rows_smem(P);
  if (smem_c > kSmemLimit || smem_r > kSmemLimit) return CVB_ERR_UNSUPPORTED_SIZE;
  const bool sy = small_axis(P.ay), sx = small_axis(P.ax);
  P.ws = (float2*)workspace;
  P.status = status_ptr();
  for (int p0 = 0; p0 < planes; p0 += r.chunk) {
    P.plane0 = p0;
    P.nplane = planes - p0 < r.chunk ? planes - p0 : r.chunk;
    if (P.s > 1)
      P.r = P.rsave ? P.rsave + (size_t)p0 * P.h * P.wp
                    : (float*)((char*)workspace + (size_t)P.nplane * P.hh * P.wp * sizeof(float2));
    const int gc = (P.nplane * P.wc + kLines - 1) / kLines, gr = (P.nplane * P.hh + kLines - 1) / kLines;
    const int tc = strip_threads(P, false, gc, sm_count()), tr = strip_threads(P, true, gr, sm_count());
    int rc = takes_fix(P, 0, sm_count()) ? launch_fix(0, P, io_dtype, sm_count(), st)
             : P.ay.mp ? matrix_entry(P.ay.mp).cols_fwd(P, io_dtype, tc, gc, smem_c, st)
             : f32   ? launch_cols_fwd_f32(P, sy, tc, gc, smem_c, st)
                     : launch_cols_fwd_bf16(P, sy, tc, gc, smem_c, st);
    if (rc == CVB_OK)
      rc = takes_fix(P, 1, sm_count()) ? launch_fix(1, P, io_dtype, sm_count(), st)
           : P.ax.mp ? matrix_entry(P.ax.mp).rows(P, io_dtype, tr, gr, smem_r, st) : launch_rows(P, sx, tr, gr, smem_r, st);
    if (rc == CVB_OK)
      rc = takes_fix(P, 2, sm_count()) ? launch_fix(2, P, io_dtype, sm_count(), st)
           : P.ay.mp ? matrix_entry(P.ay.mp).cols_inv(P, io_dtype, tc, gc, smem_c, st)
           : f32   ? launch_cols_inv_f32(P, sy, tc, gc, smem_c, st)
                   : launch_cols_inv_bf16(P, sy, tc, gc, smem_c, st);
    if (rc == CVB_OK && P.s > 1) rc = f32 ? launch_epilogue_f32(P, st) : launch_epilogue_bf16(P, st);
    if (rc != CVB_OK) return rc;
  }
  return CVB_OK;
}

}  // namespace rp
}  // namespace cvb
