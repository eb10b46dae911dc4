// Gradients of the Converse2D solve with the stages of cvb_rp.cuh.
//
// With y = pad(x), out = crop(solve(y)) linear in y and g = dL/dout:
//   scale 1   q = g extended by zeros to the padded plane
//   scale s   q[m] = sum_a K[a] g_full[s m - a + c]   (adjoint of corr(K, zero_insert(.)), adjoint_epilogue_body)
//   dL/dy     = IFFT2( conj(M) FFT2(q) )  (+ the cell sums of g at scale s);  dL/dx = adjoint of the padding
//   dL/dM     through  D[f] = sum over the batch of FFT2(y)[f] conj(FFT2(q)[f]),  L = Re sum M D / (h w)
// FFT2(y) and FFT2(q) meet in one kernel (rows_bwd_body): a block owns 16 rows of one channel, walks over its part of
// the batch, transforms both planes' rows, adds their products to an accumulator tile and sends the second on through
// the conjugated multiplier -- D costs no transform of its own and no atomics.  The chain rule from D to the k x k taps
// and lambda is closed form (chain_body); the taps also enter the epilogue's correlation directly (tap sums of
// adjoint_epilogue_body).
#pragma once
#include "cvb_rp.cuh"

namespace cvb {
namespace rp {

struct BwdParams {
  Params P;               // geometry, table; ws = row spectra of q
  const float2* wx;       // row spectra of y: [B C][hh][wp]
  float2* D;              // [nseg][C][w][hh], four times the sum over the segment's batch entries
  int nseg;
  int solve;              // 0: only D is wanted (q is not sent on)
};

// 16 rows from global memory through the R0-point transforms into a tile
template <int MAXR, int MP>
__device__ __forceinline__ void rows_first(const Params& P, const float2* W, float2* T, const float* mats, int nl) {
  const int tid = threadIdx.x, nthr = blockDim.x, pitch = P.pitch;
  const Axis& ax = P.ax;
  const int r0 = ax.r0, r1 = ax.r1;
  if constexpr (MP == 0) {
    dispatch<MAXR>(r0, [&](auto ic) {
      constexpr int R = decltype(ic)::value;
      for (int it = tid; it < nl * r1; it += nthr) {
        int row, j;
        divmod_small(it, r1, ax.inv_r1, row, j);
        const float2* src = W + (size_t)row * P.wp + j;
        float re[R], im[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
          const float2 v = src[r1 * q];
          re[q] = v.x; im[q] = v.y;
        }
        Radix<R>::fwd(re, im);
        float2* dst = T + row * pitch + j;
#pragma unroll
        for (int k = 0; k < R; ++k) dst[k * r1] = make_float2(re[k], im[k]);
      }
    });
  } else {
    for (int row = tid >> 5; row < nl; row += nthr >> 5) {
      const float2* src = W + (size_t)row * P.wp;
      for (int x = tid & 31; x < P.w; x += 32) T[row * pitch + x] = src[x];
    }
    __syncthreads();
    matrix_stage<MP>(r0, r1 << kLinesLog2, r1, mats,
                     [&](int v) { return T + (v & (kLines - 1)) * pitch + (v >> kLinesLog2); });
  }
}

// spectra of y and q at position k0 of a row (R1 frequencies): D += X conj(Q), q -> conj(M) q, back to the tile
template <int R>
__device__ __forceinline__ void rows_bwd_mid(const Params& P, float (&xr)[R], float (&xi)[R], float (&qr)[R],
                                             float (&qi)[R], float2* Dk, float2* Qk, const float2* tab, int k0, int solve) {
  const Axis& ax = P.ax;
  const float2* tw = ax.tw + k0 * ax.r1;
  twiddle<R>(xr, xi, tw);
  Radix<R>::fwd(xr, xi);
  twiddle<R>(qr, qi, tw);
  Radix<R>::fwd(qr, qi);
#pragma unroll
  for (int j = 0; j < R; ++j) {
    float2 d = Dk[j];
    d.x = fmaf(xr[j], qr[j], fmaf(xi[j], qi[j], d.x));
    d.y = fmaf(xi[j], qr[j], fmaf(-xr[j], qi[j], d.y));
    Dk[j] = d;
  }
  if (!solve) return;
  const size_t ts = (size_t)ax.r0 * P.hh;
  const float2* tp = tab + (size_t)k0 * P.hh;
#pragma unroll
  for (int j = 0; j < R; ++j) {
    const float2 g = __ldg(tp + j * ts);
    const float a = qr[j], b = qi[j];
    qr[j] = fmaf(b, g.y, a * g.x);         // conj(q conj(M))
    qi[j] = fmaf(a, g.y, -b * g.x);
  }
  Radix<R>::fwd(qr, qi);
  twiddle<R>(qr, qi, tw);
#pragma unroll
  for (int j = 0; j < R; ++j) Qk[j] = make_float2(qr[j], qi[j]);
}

// grid (row groups, channels, batch segments); shared memory: three tiles of 16 rows, the matrices
template <int MAXR, int MP>
__device__ __forceinline__ void rows_bwd_body(const BwdParams& Q, float2* sm) {
  const Params& P = Q.P;
  const int tid = threadIdx.x, nthr = blockDim.x, pitch = P.pitch;
  constexpr int sh = kLinesLog2, NL = kLines;
  const Axis& ax = P.ax;
  const int r0 = ax.r0, r1 = ax.r1, tile = (pitch * NL + 1) & ~1;
  float2 *TX = sm, *TG = sm + tile, *DA = sm + 2 * tile;
  float* mats = (float*)(sm + 3 * tile);
  const int k_0 = blockIdx.x * NL, c = blockIdx.y, seg = blockIdx.z;
  const int nl = P.hh - k_0 < NL ? P.hh - k_0 : NL;
  if constexpr (MP > 0) copy_matrices<MP>(mats, ax);
  for (int i = tid; i < pitch * NL; i += nthr) DA[i] = make_float2(0.f, 0.f);
  const int row = tid & (NL - 1);
  const float2* tab = P.tab + (size_t)c * P.w * P.hh + k_0 + row;
  for (int b = seg; b < P.B; b += Q.nseg) {
    const size_t off = ((size_t)(b * P.C + c) * P.hh + k_0) * P.wp;
    float2* W = P.ws + off;
    rows_first<MAXR, MP>(P, Q.wx + off, TX, mats, nl);
    rows_first<MAXR, MP>(P, W, TG, mats, nl);
    __syncthreads();
    if (row < nl) {
      float2 *x = TX + row * pitch, *g = TG + row * pitch, *d = DA + row * pitch;
      dispatch<MAXR>(r1, [&](auto ic) {
        constexpr int R = decltype(ic)::value;
        if constexpr (MP == 0) {
          for (int k0 = tid >> sh; k0 < r0; k0 += nthr >> sh) {
            float xr[R], xi[R], qr[R], qi[R];
#pragma unroll
            for (int j = 0; j < R; ++j) {
              const float2 u = x[k0 * r1 + j], v = g[k0 * r1 + j];
              xr[j] = u.x; xi[j] = u.y; qr[j] = v.x; qi[j] = v.y;
            }
            rows_bwd_mid<R>(P, xr, xi, qr, qi, d + k0 * r1, g + k0 * r1, tab, k0, Q.solve);
          }
        } else {
          // positions kk and r0 - kk share what they read: both by one thread, the second kept in the tile's cells
          for (int kk = tid >> sh; kk <= r0 / 2; kk += nthr >> sh) {
            const bool self = kk == 0 || 2 * kk == r0;
            float2 *g0 = g + kk * r1, *g1 = g + (r0 - kk) * r1;
            const float2 *x0 = x + kk * r1, *x1 = x + (r0 - kk) * r1;
            float hr[R], hi[R];        // q at the mirrored position
            float xr[R], xi[R], qr[R], qi[R];
#pragma unroll
            for (int j = 0; j < R; ++j) {
              const float2 a = g0[j], e = self ? make_float2(0.f, 0.f) : g1[j];
              qr[j] = a.x + e.y; qi[j] = a.y - e.x;
              hr[j] = a.x - e.y; hi[j] = a.y + e.x;
              const float2 u = x0[j], v = self ? make_float2(0.f, 0.f) : x1[j];
              xr[j] = u.x + v.y; xi[j] = u.y - v.x;
            }
            rows_bwd_mid<R>(P, xr, xi, qr, qi, d + kk * r1, g0, tab, kk, Q.solve);
            if (!self) {
#pragma unroll
              for (int j = 0; j < R; ++j) {
                const float2 u = x0[j], v = x1[j];
                xr[j] = u.x - v.y; xi[j] = u.y + v.x;
              }
              rows_bwd_mid<R>(P, xr, xi, hr, hi, d + (r0 - kk) * r1, g1, tab, r0 - kk, Q.solve);
            }
          }
        }
      });
    }
    __syncthreads();
    if (Q.solve) {
      if constexpr (MP == 0) {
        dispatch<MAXR>(r0, [&](auto ic) {
          constexpr int R = decltype(ic)::value;
          for (int it = tid; it < nl * r1; it += nthr) {
            int rw, j;
            divmod_small(it, r1, ax.inv_r1, rw, j);
            const float2* src = TG + rw * pitch + j;
            float re[R], im[R];
#pragma unroll
            for (int q = 0; q < R; ++q) {
              const float2 v = src[r1 * q];
              re[q] = v.x; im[q] = v.y;
            }
            Radix<R>::fwd(re, im);
            float2* dst = W + (size_t)rw * P.wp + j;
#pragma unroll
            for (int k = 0; k < R; ++k) dst[k * r1] = make_float2(re[k], im[k]);
          }
        });
      } else {
        matrix_stage<MP>(r0, r1 << sh, r1, mats, [&](int v) { return TG + (v & (NL - 1)) * pitch + (v >> sh); });
        __syncthreads();
        for (int rw = tid >> 5; rw < nl; rw += nthr >> 5) {
          float2* dst = W + (size_t)rw * P.wp;
          for (int x = tid & 31; x < P.w; x += 32) {
            int q, j;
            divmod_small(x, r1, ax.inv_r1, q, j);
            dst[x] = matrix_value(TG + rw * pitch + j, r0, q, r1);
          }
        }
      }
      __syncthreads();
    }
  }
  __syncthreads();
  if (row < nl) {
    float2* out = Q.D + (size_t)(seg * P.C + c) * P.w * P.hh + k_0 + row;
    for (int i = tid >> sh; i < P.w; i += nthr >> sh) {   // position i = k0 r1 + j2: frequency k0 + r0 j2
      int k0, j2;
      divmod_small(i, r1, ax.inv_r1, k0, j2);
      out[(size_t)(k0 + r0 * j2) * P.hh] = DA[row * pitch + i];
    }
  }
}

// ------------------------------------------------------------------ adjoint of the upsampling epilogue
struct AdjointParams {
  const float* g;         // (B,C,sH,sW)
  const float* r;         // [B C][h][wp], or null (no tap sums wanted)
  const float* weight;    // (C,k,k)
  float* v;               // (B,C,h,w)
  float* taps;            // [B C][k k]
  int C, H, W, k, s, p, h, w, wp;
};
// One block per plane.  A thread owns two neighbouring cells at a time; the (k + s) x k window of g that they share is
// read once, row by row, and serves both the correlation and the tap products.
template <int K, int S>
__device__ __forceinline__ void adjoint_epilogue_body(const AdjointParams& A, float* red) {
  const int tid = threadIdx.x, nthr = blockDim.x, plane = blockIdx.x, ch = plane % A.C;
  constexpr int c = K / 2, NW = K + S;
  const int sH = S * A.H, sW = S * A.W, sh = S * A.h, sw = S * A.w, off = S * A.p;
  const float* g = A.g + (size_t)plane * sH * sW;
  float kw[K * K], acc[K * K];
#pragma unroll
  for (int i = 0; i < K * K; ++i) { kw[i] = A.weight[(size_t)ch * K * K + i]; acc[i] = 0.f; }
  const int pairs = (A.w + 1) / 2, total = A.h * pairs;
  const float inv = 1.0f / (float)pairs;
  // the window of a pair of cells starts (c - K + 1) mod 4 past a multiple of four columns: three 16-byte loads a row
  constexpr int SHIFT = ((c - K + 1) % 4 + 4) % 4, NV = (SHIFT + NW + 3) / 4;
  const bool quads = S % 2 == 0 && off % 4 == 0 && sW % 4 == 0 && ((size_t)A.g) % 16 == 0;
  for (int it = tid; it < total; it += nthr) {
    int my, px;
    divmod_small(it, pairs, inv, my, px);
    const int mx = 2 * px;
    const bool two = mx + 1 < A.w;
    float r0 = 0.f, r1 = 0.f;
    if (A.r) {
      const float2 rr = *(const float2*)(A.r + ((size_t)plane * A.h + my) * A.wp + mx);
      r0 = rr.x;
      if (two) r1 = rr.y;
    }
    // columns S mx + S + c - i, i = 0 .. NW - 1 (the second cell starts S to the right)
    int gx[NW];
#pragma unroll
    for (int i = 0; i < NW; ++i) {
      int x = S * mx + S + c - i;
      x = x < 0 ? x + sw : x >= sw ? x - sw : x;
      x -= off;
      gx[i] = (unsigned)x < (unsigned)sW ? x : -1;
    }
    const int lo = S * mx + c - K + 1 - off - SHIFT;    // first loaded column of the fast path
    const bool fast = quads && lo >= 0 && lo + 4 * NV <= sW;
    float v0 = 0.f, v1 = 0.f;
#pragma unroll
    for (int a = 0; a < K; ++a) {
      int y = S * my - a + c;
      y = y < 0 ? y + sh : y >= sh ? y - sh : y;
      y -= off;
      if ((unsigned)y >= (unsigned)sH) continue;
      const float* row = g + (size_t)y * sW;
      float win[NW];                                    // win[i]: column S mx + S + c - i
      if (fast) {
        float q[4 * NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          const float4 t = __ldg((const float4*)(row + lo) + i);
          q[4 * i] = t.x; q[4 * i + 1] = t.y; q[4 * i + 2] = t.z; q[4 * i + 3] = t.w;
        }
#pragma unroll
        for (int i = 0; i < NW; ++i) win[i] = q[SHIFT + NW - 1 - i];
      } else {
#pragma unroll
        for (int i = 0; i < NW; ++i) win[i] = gx[i] >= 0 ? row[gx[i]] : 0.f;
      }
#pragma unroll
      for (int b = 0; b < K; ++b) {
        v0 = fmaf(kw[a * K + b], win[S + b], v0);
        v1 = fmaf(kw[a * K + b], win[b], v1);
        acc[a * K + b] = fmaf(win[S + b], r0, fmaf(win[b], r1, acc[a * K + b]));
      }
    }
    float* o = A.v + ((size_t)plane * A.h + my) * A.w + mx;
    o[0] = v0;
    if (two) o[1] = v1;
  }
  if (!A.taps) return;
#pragma unroll
  for (int t = 0; t < K * K; ++t) {
    float x = acc[t];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if ((tid & 31) == 0) red[(tid >> 5) * K * K + t] = x;
  }
  __syncthreads();
  for (int t = tid; t < K * K; t += nthr) {
    float x = 0.f;
    for (int i = 0; i < nthr / 32; ++i) x += red[i * K * K + t];
    A.taps[(size_t)plane * K * K + t] = x;
  }
}
// any tap count and scale
__device__ __forceinline__ void adjoint_epilogue_any(const AdjointParams& A, float* red) {
  const int tid = threadIdx.x, nthr = blockDim.x, plane = blockIdx.x, ch = plane % A.C;
  const int k = A.k, s = A.s, c = k / 2, sH = s * A.H, sW = s * A.W, sh = s * A.h, sw = s * A.w, off = s * A.p;
  const float* g = A.g + (size_t)plane * sH * sW;
  const float* K = A.weight + (size_t)ch * k * k;
  auto at = [&](int my, int mx, int a, int b) {
    int y = s * my - a + c, x = s * mx - b + c;
    y = y < 0 ? y + sh : y >= sh ? y - sh : y;
    x = x < 0 ? x + sw : x >= sw ? x - sw : x;
    y -= off; x -= off;
    return (unsigned)y < (unsigned)sH && (unsigned)x < (unsigned)sW ? g[(size_t)y * sW + x] : 0.f;
  };
  for (int i = tid; i < A.h * A.w; i += nthr) {
    const int my = i / A.w, mx = i - my * A.w;
    float v = 0.f;
    for (int a = 0; a < k; ++a)
      for (int b = 0; b < k; ++b) v = fmaf(K[a * k + b], at(my, mx, a, b), v);
    A.v[(size_t)plane * A.h * A.w + i] = v;
  }
  if (!A.taps) return;
  for (int t = 0; t < k * k; ++t) {
    float x = 0.f;
    for (int i = tid; i < A.h * A.w; i += nthr) {
      const int my = i / A.w, mx = i - my * A.w;
      x = fmaf(at(my, mx, t / k, t % k), A.r[((size_t)plane * A.h + my) * A.wp + mx], x);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if ((tid & 31) == 0) red[tid >> 5] = x;
    __syncthreads();
    if (tid == 0) {
      float y = 0.f;
      for (int i = 0; i < nthr / 32; ++i) y += red[i];
      A.taps[(size_t)plane * k * k + t] = y;
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------ adjoint of the padding (+ cell sums of g)
struct PadAdjointParams {
  const float* f;         // (B,C,h,w)
  const float* g;         // (B,C,sH,sW) at scale s >= 2, else null
  float* gx;              // (B,C,H,W)
  int H, W, s, p, h, w, pad_mode;
};
// padded indices that read source index i of an axis of length n: a run [first, last] and up to two single ones
struct Preimage { int first, last, e0, e1; };
__device__ __forceinline__ Preimage preimage(int i, int n, int p, int mode) {
  Preimage r = {i + p, i + p, -1, -1};
  if (mode == 0) {                                   // circular: copies n to the left and to the right
    if (i >= n - p) r.e0 = i + p - n;
    if (i < p) r.e1 = i + p + n;
  } else if (mode == 1) {                            // replicate: the edges stand for the whole margin
    if (i == 0) r.first = 0;
    if (i == n - 1) r.last = n + 2 * p - 1;
  } else if (mode == 2) {                            // reflect
    if (i >= 1 && i <= p) r.e0 = p - i;
    if (i <= n - 2 && i >= n - 1 - p) r.e1 = 2 * n - 2 - i + p;
  }
  return r;
}
__device__ __forceinline__ float pad_adjoint_at(const PadAdjointParams& A, const float* f, int y, int x) {
  // away from the margins' images a source sample has one padded copy
  if (y > A.p && y < A.H - 1 - A.p && x > A.p && x < A.W - 1 - A.p) return f[(size_t)(y + A.p) * A.w + x + A.p];
  const Preimage py = preimage(y, A.H, A.p, A.pad_mode), px = preimage(x, A.W, A.p, A.pad_mode);
  auto row = [&](int yy) {
    const float* q = f + (size_t)yy * A.w;
    float t = 0.f;
    for (int xx = px.first; xx <= px.last; ++xx) t += q[xx];
    if (px.e0 >= 0) t += q[px.e0];
    if (px.e1 >= 0) t += q[px.e1];
    return t;
  };
  float v = 0.f;
  for (int yy = py.first; yy <= py.last; ++yy) v += row(yy);
  if (py.e0 >= 0) v += row(py.e0);
  if (py.e1 >= 0) v += row(py.e1);
  return v;
}
__device__ __forceinline__ void pad_adjoint_body(const PadAdjointParams& A) {
  const int plane = blockIdx.y;
  const float* f = A.f + (size_t)plane * A.h * A.w;
  float* out = A.gx + (size_t)plane * A.H * A.W;
  const int start = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  if (A.g && A.s == 2 && A.W % 2 == 0 && ((size_t)A.g) % 16 == 0 && ((size_t)A.gx) % 8 == 0) {
    // two samples at a time: their eight values of g are two 16-byte loads
    const int half = A.W / 2;
    const float inv = 1.0f / (float)half;
    const float* g = A.g + (size_t)plane * 4 * A.H * A.W;
    for (int i = start; i < A.H * half; i += step) {
      int y, xh;
      divmod_small(i, half, inv, y, xh);
      const float4 a = __ldg((const float4*)(g + (size_t)(2 * y) * 2 * A.W) + xh);
      const float4 b = __ldg((const float4*)(g + (size_t)(2 * y + 1) * 2 * A.W) + xh);
      const float v0 = pad_adjoint_at(A, f, y, 2 * xh) + ((a.x + a.y) + (b.x + b.y));
      const float v1 = pad_adjoint_at(A, f, y, 2 * xh + 1) + ((a.z + a.w) + (b.z + b.w));
      ((float2*)out)[i] = make_float2(v0, v1);
    }
    return;
  }
  const float invW = 1.0f / (float)A.W;
  for (int i = start; i < A.H * A.W; i += step) {
    int y, x;
    divmod_small(i, A.W, invW, y, x);
    float v = pad_adjoint_at(A, f, y, x);
    if (A.g) {
      const float* g = A.g + ((size_t)plane * A.s * A.H + (size_t)A.s * y) * A.s * A.W + A.s * x;
      for (int a = 0; a < A.s; ++a)
        for (int b = 0; b < A.s; ++b) v += g[(size_t)a * A.s * A.W + b];
    }
    out[i] = v;
  }
}

}  // namespace rp
}  // namespace cvb
