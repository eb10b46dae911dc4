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
#include "cvb_fix.cuh"
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
  int tw, th, nx, ny, pitch;     // plan_adjoint: a tile is th x tw items of 2 x 2 cells
  float inv_tw;
};
// One block per plane walks over tiles of it: the part of g that a tile's cells read, wrapped and extended by zeros, and r are
// copied to shared memory asynchronously while the previous tile is worked on.  A thread owns 2 x 2 neighbouring cells; the
// (K + s) x (K + s) window that they share is read row by row, 16 bytes at a time (two cells apart: no bank conflicts at
// scale 2), and serves both the correlation and the tap products, two columns an instruction.  1024 planes of 68 x 68, scale
// 2, 5 x 5 taps: 43 us, issue slots 62 % busy, the port to shared memory 56 %, 17 % of the blocks' time the third, short wave;
// 105 MB take 16 us.  With rows of g loaded by each thread as it needed them, one row's latency after the other: 112 us.
// Tried: taps in registers and two blocks an SM 59 us; without the packed products 55 (copies indexed chunk by chunk in both).
template <int K, int S>
struct AdjointTile {
  static constexpr int c = K / 2, NW = K + S, SHIFT = ((c - K + 1) % 4 + 4) % 4, NV = (SHIFT + NW + 3) / 4;
  // Blocks of an SM: three leave a thread 80 registers, which up to five taps a side take with 24 bytes spilled at most; at scale
  // 4 five taps would spill 64 bytes and seven taps 356 to 496 at any scale (none and 40 to 56 with 128 registers).  `area`: bytes
  // that a block's two tiles may take.
  static constexpr int threads = 256, sums = threads + 8, blocks = K < 7 && K * S < 20 ? 3 : 2, area = 216 * 1024 / blocks;
  __host__ __device__ static int rows(int th) { return 2 * S * th + K - S; }
  __host__ __device__ static int floats(const AdjointParams& A) {
    const int t = 2 * buffer(A), red = K * K * sums;
    return taps + (t > red ? t : red);
  }
  // Taps in ascending order of the columns that they meet, two at a time where the window has them in one aligned pair:
  // LEAD alone, NP pairs, TAIL alone; in shared memory rows of KP, the pairs aligned
  static constexpr int LEAD = SHIFT & 1, NP = (K - LEAD) / 2, TAIL = (K - LEAD) & 1, KP = (K + LEAD + 3) & ~3, taps = K * KP;
  // g's part of a tile, then r's
  __host__ __device__ static int buffer(const AdjointParams& A) { return rows(A.th) * A.pitch + 4 * A.th * A.tw; }
};
// At most 64 items side by side (524 floats a row at scale 4: two tiles of one item's rows always fit); as many rows of items
// as make the walk shortest by a rough count of a block's cycles -- 520 for every 256 items, 15 floats copied per cycle, 150
// a tile -- as fit 36 KB a tile where three blocks share an SM, 54 KB where two do.
template <int K, int S>
inline void plan_adjoint(AdjointParams& A) {
  using T = AdjointTile<K, S>;
  const int cols = (A.w + 1) / 2, lines = (A.h + 1) / 2;
  A.nx = (cols + 63) / 64;
  A.tw = ((cols + A.nx - 1) / A.nx + 1) & ~1;          // even: tiles start at a multiple of four columns at every scale
  A.pitch = (2 * S * A.tw - S + K + T::SHIFT + S + 3) & ~3;
  if (A.pitch < 2 * S * (A.tw - 1) + 4 * T::NV) A.pitch = (2 * S * (A.tw - 1) + 4 * T::NV + 3) & ~3;
  A.inv_tw = 1.0f / (float)A.tw;
  long long best = -1;
  for (int th = 1; th <= lines; ++th) {
    const int area = T::rows(th) * A.pitch + 4 * th * A.tw;
    if (th > 1 && 8 * area > T::area) break;
    const long long cost = (long long)((lines + th - 1) / th) *
        ((th * A.tw + T::threads - 1) / T::threads * 520 + area / 15 + 150);
    if (best < 0 || cost < best) { best = cost; A.th = th; }
  }
  A.ny = (lines + A.th - 1) / A.th;
}
template <int K, int S>
__device__ __forceinline__ void adjoint_epilogue_body(const AdjointParams& A, float* sm) {
  using T = AdjointTile<K, S>;
  constexpr int c = T::c, NW = T::NW, SHIFT = T::SHIFT, NV = T::NV;
  const int tid = threadIdx.x, nthr = blockDim.x, plane = blockIdx.x, ch = plane % A.C;
  const int sH = S * A.H, sW = S * A.W, sh = S * A.h, sw = S * A.w, off = S * A.p;
  const float* g = A.g + (size_t)plane * sH * sW;
  const int nrow = T::rows(A.th), size = T::buffer(A), ntile = A.nx * A.ny;
  float *kw = sm, *tiles = sm + T::taps;
  // 16-byte copies where the columns of g and of the tile agree modulo 4
  const bool quads = off % 4 == 0 && sW % 4 == 0 && (size_t)A.g % 16 == 0;
  // a thread copies 16 bytes of every gstep-th row of a tile of g and 8 of every rstep-th row of r
  const int chunks = A.pitch / 4, gj = tid / chunks, gq = tid - gj * chunks, gstep = nthr / chunks;
  const int rj = tid / A.tw, rq = tid - rj * A.tw, rstep = nthr / A.tw;
  auto load = [&](int t) {
    float *buf = tiles + (t & 1) * size, *rbuf = buf + nrow * A.pitch;
    const int ty = t / A.nx, cy = 2 * A.th * ty, cx = 2 * A.tw * (t - ty * A.nx);      // the tile's first cell
    const int y0 = S * cy + c - K + 1, x0 = S * cx + c - K + 1 - SHIFT;
    auto wrapped = [&](int i, int n) { return (i < 0 ? i + n : i >= n ? i - n : i) - off; };
    if (quads) {     // the period is a multiple of four columns too: four columns are in g or not, together
      const int x = wrapped(x0 + 4 * gq, sw);
      const bool in = gj < gstep && (unsigned)x < (unsigned)sW;
      const float* src = g + (in ? x : 0);
      float* dst = buf + gj * A.pitch + 4 * gq;
#pragma unroll 1
      for (int j = gj < gstep ? gj : nrow; j < nrow; j += gstep, dst += gstep * A.pitch) {
        const int y = wrapped(y0 + j, sh), near = y < 0 ? 0 : y < sH ? y : sH - 1;
        fx_copy<16>(dst, src + (size_t)near * sW, in && y == near);
      }
    } else {
      for (int i = tid & 31; i < A.pitch; i += 32) {
        const int x = wrapped(x0 + i, sw);
        const bool in = (unsigned)x < (unsigned)sW;
        const float* src = g + (in ? x : 0);
#pragma unroll 1
        for (int j = tid >> 5; j < nrow; j += nthr >> 5) {
          const int y = wrapped(y0 + j, sh), near = y < 0 ? 0 : y < sH ? y : sH - 1;
          fx_copy<4>(buf + j * A.pitch + i, src + (size_t)near * sW, in && y == near);
        }
      }
    }
    if (!A.r) return;
    const bool in = cx + 2 * rq < A.w;
    const float* src = A.r + ((size_t)plane * A.h + cy) * A.wp + (in ? cx + 2 * rq : 0);
    const int have = A.h - cy;
#pragma unroll 1
    for (int j = rj < rstep ? rj : 2 * A.th; j < 2 * A.th; j += rstep)
      fx_copy<8>(rbuf + 2 * (A.tw * j + rq), src + (j < have ? j : 0) * A.wp, in && j < have);
  };
  constexpr int LEAD = T::LEAD, NP = T::NP, TAIL = T::TAIL, KP = T::KP;
  float2 acc[K][NP];
  float lead[K], tail[K];
#pragma unroll
  for (int a = 0; a < K; ++a) {
    lead[a] = tail[a] = 0.f;
#pragma unroll
    for (int i = 0; i < NP; ++i) acc[a][i] = make_float2(0.f, 0.f);
  }
  for (int i = tid; i < K * K; i += nthr) {
    const int a = i / K, b = i - a * K;
    kw[a * KP + LEAD + K - 1 - b] = A.weight[(size_t)ch * K * K + i];
  }
  load(0);
  for (int t = 0; t < ntile; ++t) {
    fx_copies_done();
    __syncthreads();                       // this tile is there, and every thread is done with the other buffer
    if (t + 1 < ntile) load(t + 1);
    const float* buf = tiles + (t & 1) * size;
    const int ty = t / A.nx, tx = t - ty * A.nx;
    for (int it = tid; it < A.th * A.tw; it += nthr) {
      int iy, ix;
      divmod_small(it, A.tw, A.inv_tw, iy, ix);
      const int my = 2 * (A.th * ty + iy), mx = 2 * (A.tw * tx + ix);
      if (my >= A.h || mx >= A.w) continue;
      const bool right = mx + 1 < A.w, below = my + 1 < A.h;
      float r[2][2] = {};
      float2 v[2][2] = {};                   // sums over the even and the odd columns
      if (A.r) {
        const float* rp = buf + nrow * A.pitch + 4 * A.tw * iy + 2 * ix;
        const float2 r0 = *(const float2*)rp, r1 = *(const float2*)(rp + 2 * A.tw);
        r[0][0] = r0.x; r[1][0] = r1.x;
        if (right) { r[0][1] = r0.y; r[1][1] = r1.y; }
      }
      const float* src = buf + 2 * S * (iy * A.pitch + ix);
#pragma unroll
      for (int j = 0; j < K + S; ++j) {
        float q[4 * NV];                   // row S my + c - K + 1 + j from column S mx + c - K + 1 - SHIFT on
        if constexpr (S % 2 == 0) {
#pragma unroll
          for (int i = 0; i < NV; ++i) {
            const float4 f = *(const float4*)(src + j * A.pitch + 4 * i);
            q[4 * i] = f.x; q[4 * i + 1] = f.y; q[4 * i + 2] = f.z; q[4 * i + 3] = f.w;
          }
        } else {
#pragma unroll
          for (int i = SHIFT; i < SHIFT + NW; ++i) q[i] = src[j * A.pitch + i];
        }
#pragma unroll
        for (int d = 0; d < 2; ++d) {      // the upper and the lower two cells
          const int a = K - 1 - j + S * d;
          if (a < 0 || a >= K) continue;
          const float* ka = kw + a * KP;
#pragma unroll
          for (int x = 0; x < 2; ++x) {    // the left and the right one
            const float* w = q + SHIFT + S * x;
            const float2 rr = make_float2(r[d][x], r[d][x]);
#pragma unroll
            for (int i = 0; i < NP; ++i) {
              const float2 f = make_float2(w[LEAD + 2 * i], w[LEAD + 2 * i + 1]);
              v[d][x] = fx_fma2(*(const float2*)(ka + 2 * LEAD + 2 * i), f, v[d][x]);
              acc[a][i] = fx_fma2(f, rr, acc[a][i]);
            }
            if constexpr (LEAD != 0) {
              v[d][x].y = fmaf(ka[1], w[0], v[d][x].y);
              lead[a] = fmaf(w[0], r[d][x], lead[a]);
            }
            if constexpr (TAIL != 0) {
              v[d][x].x = fmaf(ka[LEAD + K - 1], w[K - 1], v[d][x].x);
              tail[a] = fmaf(w[K - 1], r[d][x], tail[a]);
            }
          }
        }
      }
      float* o = A.v + ((size_t)plane * A.h + my) * A.w + mx;
#pragma unroll
      for (int d = 0; d < 2; ++d) {
        if (d && !below) break;
        if (right && A.w % 2 == 0) *(float2*)(o + d * A.w) = make_float2(v[d][0].x + v[d][0].y, v[d][1].x + v[d][1].y);
        else {
          o[d * A.w] = v[d][0].x + v[d][0].y;
          if (right) o[d * A.w + 1] = v[d][1].x + v[d][1].y;
        }
      }
    }
  }
  if (!A.taps) return;
  __syncthreads();
#pragma unroll
  for (int t = 0; t < K * K; ++t) {
    const int a = t / K, e = K - 1 - (t - a * K) - LEAD;
    tiles[t * T::sums + tid] = e < 0 ? lead[a] : e == 2 * NP ? tail[a] : e % 2 ? acc[a][e / 2].y : acc[a][e / 2].x;
  }
  __syncthreads();
  for (int t0 = 0; t0 < K * K; t0 += nthr / 8) {          // eight threads a tap
    const int t = t0 + (tid >> 3);
    float x = 0.f;
    if (t < K * K)
      for (int i = tid & 7; i < nthr; i += 8) x += tiles[t * T::sums + i];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (t < K * K && (tid & 7) == 0) A.taps[(size_t)plane * K * K + t] = x;
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
__device__ __forceinline__ float cell_sum(const PadAdjointParams& A, const float* g, int y, int x) {
  const float* q = g + ((size_t)A.s * A.W * y + x) * A.s;
  if (A.s == 2) {
    const float *lo = q, *hi = q + 2 * A.W;
    return (lo[0] + lo[1]) + (hi[0] + hi[1]);
  }
  float v = 0.f;
  for (int a = 0; a < A.s; ++a)
    for (int b = 0; b < A.s; ++b) v += q[(size_t)a * A.s * A.W + b];
  return v;
}
// Bounds: the latency of the loads (f, g and gx once each).  Samples away from the margins' images have one padded copy: a thread does
// four of them with all loads in flight.  The others -- 18 % of a 64 x 64 plane at p = 2, 39 % at p = 6 -- are numbered
// by themselves (top and bottom bands, then the left and right ends of the rows between), so that the lanes of a warp that
// walk through their copies all have copies to walk through.
constexpr int kPadAdjointUnroll = 4;
__device__ __forceinline__ void pad_adjoint_body(const PadAdjointParams& A) {
  const int plane = blockIdx.y;
  const float* f = A.f + (size_t)plane * A.h * A.w;
  const float* g = A.g ? A.g + (size_t)plane * A.s * A.H * A.s * A.W : nullptr;
  float* out = A.gx + (size_t)plane * A.H * A.W;
  const int start = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  const int m = A.p + 1;                                  // y <= p or y >= H - 1 - p: may have further copies
  const int ih = A.H > 2 * m ? A.H - 2 * m : 0, iw = A.W > 2 * m ? A.W - 2 * m : 0;
  const float invW = 1.0f / (float)A.W;
  auto inner = [&](int y, int x) { return y >= m && y < A.H - m && x >= m && x < A.W - m; };
  if (ih && iw) {
    const int lo = m * A.W, hi = (A.H - m) * A.W;         // rows between the bands
    if (g && A.s == 2 && A.W % 2 == 0 && (size_t)A.g % 16 == 0) {
      // two samples at a time: their eight values of g are two 16-byte loads
      const int half = A.W / 2;
      const float inv = 1.0f / (float)half;
      for (int i0 = lo / 2 + start; i0 < hi / 2; i0 += 2 * step) {
        float4 a[2], b[2];
        float2 v[2];
        int y[2], x[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int i = i0 + u * step;
          if (i >= hi / 2) continue;
          divmod_small(i, half, inv, y[u], x[u]);
          a[u] = __ldg((const float4*)(g + (size_t)(2 * y[u]) * 2 * A.W) + x[u]);
          b[u] = __ldg((const float4*)(g + (size_t)(2 * y[u] + 1) * 2 * A.W) + x[u]);
          const float* q = f + (size_t)(y[u] + A.p) * A.w + 2 * x[u] + A.p;
          v[u] = make_float2(q[0], q[1]);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int i = i0 + u * step;
          if (i >= hi / 2) continue;
          if (inner(y[u], 2 * x[u])) out[2 * i] = v[u].x + ((a[u].x + a[u].y) + (b[u].x + b[u].y));
          if (inner(y[u], 2 * x[u] + 1)) out[2 * i + 1] = v[u].y + ((a[u].z + a[u].w) + (b[u].z + b[u].w));
        }
      }
    } else {
      constexpr int U = kPadAdjointUnroll;
      for (int i0 = lo + start; i0 < hi; i0 += U * step) {
        float v[U];
        int x[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int i = i0 + u * step;
          x[u] = 0;
          if (i >= hi) continue;
          int y;
          divmod_small(i, A.W, invW, y, x[u]);
          v[u] = f[(size_t)(y + A.p) * A.w + x[u] + A.p];
          if (g && x[u] >= m && x[u] < A.W - m) v[u] += cell_sum(A, g, y, x[u]);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (x[u] >= m && x[u] < A.W - m) out[i0 + u * step] = v[u];     // x stays 0 past the end
      }
    }
  }
  const int band = ih && iw ? 2 * m * A.W : A.H * A.W, edges = band + (ih && iw ? 2 * m * ih : 0);
  for (int e = start; e < edges; e += step) {
    int y, x;
    if (e < band) {
      divmod_small(e, A.W, invW, y, x);
      if (ih && iw && y >= m) y += ih;
    } else {
      const int q = (e - band) / (2 * m), i = e - band - q * 2 * m;
      y = m + q;
      x = i < m ? i : A.W - 2 * m + i;
    }
    float v = pad_adjoint_at(A, f, y, x);
    if (g) v += cell_sum(A, g, y, x);
    out[(size_t)y * A.W + x] = v;
  }
}

}  // namespace rp
}  // namespace cvb
