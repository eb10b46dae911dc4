// The Converse2D solve on real planes, any two-stage plan chosen at run time.
//
// A real plane y (h x w, padded) is transformed alone: columns 2c and 2c+1 travel as the real and the
// imaginary part of one complex column, and after the column transform the two spectra are separated
// (E = Z[k] + conj Z[-k], O = (Z[k] - conj Z[-k]) / i, twice the spectra: the table carries the 1/2), so
// only the rows k = 0 .. h/2 are transformed along x and only half of the multiplier exists.  That is
// the work of packing two planes into one complex plane, without needing a second plane that shares
// the taps: a single image, an odd batch and per-sample kernels cost what they should.
//
//   columns forward   y -> Z[k][c] -> E, O = S^[k][x]           c < wc = ceil(w / 2), k <= h / 2
//   rows              S^ -> along x -> . table, conjugate -> along x -> U[k][x] = conj(T[k][x])
//   columns inverse   V[k] = U[k][2c] - i U[k][2c+1],  V[h - k] = conj U[k][2c] - i conj U[k][2c+1]
//                     -> forward transform -> (column 2c, -column 2c+1): crop and store, or the plane r
//                     of the upsampling form  out = nearest(y) + corr(K, zero_insert(r))
//
// Every axis is N = R0 * R1.  Forward and inverse run the same forward transform (the inverse on the
// conjugated spectrum): index j + R1 q over q (R0 points) -> k0, twiddle exp(-2 pi i k0 j / N), over j
// (R1 points) -> j2, frequency k0 + R0 j2; the way back k0 + R0 j2 over j2 -> j, twiddle, over k0 -> q.
// R1 is a register butterfly; R0 is one too (up to 32) or, for lengths with a large prime, a dense
// R0-point transform ("matrix stage", any R0 <= 127) that keeps cosine / sine rows in the table blob.
//
// Two kernels families share the stage code: one block per plane with everything in shared memory
// (plane_body), and three launches that meet in a workspace S^[plane][k][x] (cols_fwd_body,
// rows_body, cols_inv_body), whose stages read and write global memory straight from the butterflies so
// that each launch needs one or two passes through shared memory.
#pragma once
#include "cvb_kernels.cuh"

namespace cvb {
namespace rp {

struct Axis {
  int n, r0, r1;
  int nkg;              // 0: R0 is a register butterfly; else groups of 8 k of the matrix stage
  float inv_r1;
  const float2* tw;     // twiddles in position order: [k0 r1 + j] = (cos, sin)(2 pi k0 j / n)
  const float2* dm;     // matrix stage: [q = 1 ..][k < 8 nkg] (cos, sin)(2 pi q k / R0)
};

struct Params {
  const void* x;
  void* out;
  const float2* tab;    // [C][w][hh]
  const float* weight;  // (C,k,k), scale >= 2
  int B, C, H, W, k, s, p, pad_mode, gelu;
  int h, w, hh, wc, wp; // hh = h / 2 + 1 rows, wc column pairs, wp = 2 wc
  int conj;             // 1: multiply by the conjugated table (the adjoint)
  int plane0, nplane;   // planes of this launch (plane = b * C + c)
  int lsh_c, lsh_r;     // log2 of the lines per block, column / row kernels
  int vec;              // p and W even, pointers aligned: pairs of columns are loaded and stored at once
  float2* ws;           // [nplane][hh][wp]
  float* r;             // scale >= 2: [nplane][h][wp]
  int pitch;            // rows kernel / plane kernel: odd row pitch (complex) of the shared-memory rows
  float inv_wc, inv_hh;
  Axis ay, ax;
};

// groups of 8 outputs of an R0-point matrix stage; 0: R0 has a register butterfly
__host__ __device__ constexpr bool register_radix(int r) {
#define CVB_RP_X(R) r == R ||
  return CVB_RP_EACH_RADIX(CVB_RP_X) false;
#undef CVB_RP_X
}
__host__ __device__ constexpr int matrix_groups(int r0) { return register_radix(r0) ? 0 : (r0 / 2 + 1 + 7) / 8; }

// Two builds of every kernel: radices up to kSmallRadix (80 registers a thread) and all radices.
constexpr int kSmallRadix = 20, kAnyRadix = 32;

template <int R> struct IC { static constexpr int value = R; };

// f(IC<R>()) for the run-time radix r <= MAXR
template <int MAXR, class F>
__device__ __forceinline__ void dispatch(int r, F&& f) {
  switch (r) {
#define CVB_RP_X(R) case R: if constexpr (R <= MAXR) f(IC<R>()); break;
    CVB_RP_EACH_RADIX(CVB_RP_X)
#undef CVB_RP_X
    default: f(IC<1>()); break;
  }
}

__device__ __forceinline__ float2 mulc(float2 v, float2 w) {   // v * conj(w)
  return make_float2(fmaf(v.y, w.y, v.x * w.x), fmaf(-v.x, w.y, v.y * w.x));
}
// multiply elements 1 .. R-1 by the conjugated twiddles t[1 .. R-1] (position order: contiguous)
template <int R>
__device__ __forceinline__ void twiddle(float (&re)[R], float (&im)[R], const float2* t) {
  if constexpr (R % 2 == 0) {
#pragma unroll
    for (int j = 0; j < R; j += 2) {
      const float4 w = __ldg((const float4*)(t + j));
      if (j > 0) {
        const float2 v = mulc(make_float2(re[j], im[j]), make_float2(w.x, w.y));
        re[j] = v.x; im[j] = v.y;
      }
      const float2 u = mulc(make_float2(re[j + 1], im[j + 1]), make_float2(w.z, w.w));
      re[j + 1] = u.x; im[j + 1] = u.y;
    }
  } else {
#pragma unroll
    for (int j = 1; j < R; ++j) {
      const float2 v = mulc(make_float2(re[j], im[j]), __ldg(t + j));
      re[j] = v.x; im[j] = v.y;
    }
  }
}

// ------------------------------------------------------------------ matrix stage
// R-point transforms of nvec vectors: in(v, q) reads element q of vector v, put(v, k, value) takes element k.
// A thread computes 8 outputs k and their mirrors R - k of VT vectors from the sums and differences of the pairs
// (q, R - q): 4 FMAs per (k, q) and vector; the cosine / sine row of a q is the same for the whole warp and is
// read through L1.  INPLACE: put overwrites what in reads, with a block barrier between (a round covers whole
// vectors).
template <bool INPLACE, int VT, class In, class Put>
__device__ __forceinline__ void matrix_rounds(const Axis& ax, int nvec, In in, Put put) {
  const int R = ax.r0, nkg = ax.nkg, tid = threadIdx.x, nthr = blockDim.x;
  int vc = nthr / nkg;
  if (vc >= 32) vc &= ~15;
  const int want = ((nvec + VT - 1) / VT + 15) & ~15;
  if (want < vc) vc = want;
  const int kg = tid / vc, vl = tid - kg * vc;
  const int QH = (R - 1) >> 1, KH = R >> 1;
  const bool even = (R & 1) == 0;
  for (int v0 = 0; v0 < nvec; v0 += VT * vc) {
    int v[VT];
    const bool act = kg < nkg && v0 + vl < nvec;
    bool last = false;
#pragma unroll
    for (int t = 0; t < VT; ++t) {
      v[t] = v0 + vl + t * vc;
      if (v[t] >= nvec) { v[t] = v0 + vl; last = true; }   // computed twice, written once
    }
    float ar[VT][8], ai[VT][8], br[VT][8], bi[VT][8];
    if (act) {
#pragma unroll
      for (int t = 0; t < VT; ++t) {
        const float2 x0 = in(v[t], 0);
        float2 xh = make_float2(0.f, 0.f);
        if (even) xh = in(v[t], KH);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float sg = (i & 1) ? -1.f : 1.f;
          ar[t][i] = fmaf(sg, xh.x, x0.x); ai[t][i] = fmaf(sg, xh.y, x0.y);
          br[t][i] = 0.f; bi[t][i] = 0.f;
        }
      }
      const float4* d = (const float4*)(ax.dm + kg * 8);
      const int dstep = nkg * 4;
#pragma unroll 2
      for (int q = 1; q <= QH; ++q, d += dstep) {
        float pr[VT], pi[VT], mr[VT], mi[VT];
#pragma unroll
        for (int t = 0; t < VT; ++t) {
          const float2 u = in(v[t], q), w = in(v[t], R - q);
          pr[t] = u.x + w.x; pi[t] = u.y + w.y; mr[t] = u.x - w.x; mi[t] = u.y - w.y;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 c = __ldg(d + i);
#pragma unroll
          for (int t = 0; t < VT; ++t) {
            ar[t][2 * i] = fmaf(c.x, pr[t], ar[t][2 * i]);         ai[t][2 * i] = fmaf(c.x, pi[t], ai[t][2 * i]);
            br[t][2 * i] = fmaf(c.y, mr[t], br[t][2 * i]);         bi[t][2 * i] = fmaf(c.y, mi[t], bi[t][2 * i]);
            ar[t][2 * i + 1] = fmaf(c.z, pr[t], ar[t][2 * i + 1]); ai[t][2 * i + 1] = fmaf(c.z, pi[t], ai[t][2 * i + 1]);
            br[t][2 * i + 1] = fmaf(c.w, mr[t], br[t][2 * i + 1]); bi[t][2 * i + 1] = fmaf(c.w, mi[t], bi[t][2 * i + 1]);
          }
        }
      }
    }
    if (INPLACE) __syncthreads();
    if (act) {
#pragma unroll
      for (int t = 0; t < VT; ++t) {
        if (t > 0 && last && v[t] == v0 + vl) continue;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int k = kg * 8 + i;
          if (k <= KH) {
            put(v[t], k, make_float2(ar[t][i] + bi[t][i], ai[t][i] - br[t][i]));
            if (k != 0 && 2 * k != R) put(v[t], R - k, make_float2(ar[t][i] - bi[t][i], ai[t][i] + br[t][i]));
          }
        }
      }
    }
  }
}
template <bool INPLACE, class In, class Put>
__device__ __forceinline__ void matrix_stage(const Axis& ax, int nvec, In in, Put put) {
  if (nvec * ax.nkg > (int)blockDim.x) matrix_rounds<INPLACE, 2>(ax, nvec, in, put);
  else matrix_rounds<INPLACE, 1>(ax, nvec, in, put);
}

// Two adjacent padded columns of one plane: what a thread reads in every row it visits.
template <typename IO>
struct ColumnPair {
  const IO* p0;         // source column of 2c (any valid column where there is none)
  const IO* p1;
  bool z0, z1;          // the column is zero (constant padding, or past an odd width)
  bool vec;             // p1 = p0 + 1 and p0 is aligned to two elements
  __device__ __forceinline__ void set(const Params& P, const IO* xp, int c, bool valid) {
    int c0 = valid ? pad_index(2 * c - P.p, P.W, P.pad_mode) : -1;
    int c1 = valid && 2 * c + 1 < P.w ? pad_index(2 * c + 1 - P.p, P.W, P.pad_mode) : -1;
    z0 = c0 < 0; z1 = c1 < 0;
    vec = P.vec && !z0 && c1 == c0 + 1;
    p0 = xp + (z0 ? 0 : c0);
    p1 = xp + (z1 ? 0 : c1);
  }
};
// padded row -> source row * W, or -1
__device__ __forceinline__ int row_offset(const Params& P, int y) {
  const int r = pad_index(y - P.p, P.H, P.pad_mode);
  return r < 0 ? -1 : r * P.W;
}
template <int R, typename IO>
__device__ __forceinline__ void load_rows(const Params& P, const ColumnPair<IO>& cp, const int* rowoff, int j, int step,
                                          float (&re)[R], float (&im)[R]) {
  if (P.pad_mode == 3) {
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int o = rowoff[j + step * q];
      re[q] = o >= 0 && !cp.z0 ? ld_io<IO>(cp.p0, (size_t)o) : 0.f;
      im[q] = o >= 0 && !cp.z1 ? ld_io<IO>(cp.p1, (size_t)o) : 0.f;
    }
  } else if (cp.vec) {
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int o = rowoff[j + step * q];
      if constexpr (sizeof(IO) == 4) {
        const float2 v = *(const float2*)(cp.p0 + o);
        re[q] = v.x; im[q] = v.y;
      } else {
        const uint32_t v = *(const uint32_t*)(cp.p0 + o);
        re[q] = __uint_as_float(v << 16); im[q] = __uint_as_float(v & 0xffff0000u);
      }
    }
  } else {
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int o = rowoff[j + step * q];
      re[q] = ld_io<IO>(cp.p0, (size_t)o);
      im[q] = ld_io<IO>(cp.p1, (size_t)o);
    }
    if (cp.z1) {     // past an odd width
#pragma unroll
      for (int q = 0; q < R; ++q) im[q] = 0.f;
    }
  }
}

// store (column 2c, -column 2c+1) of padded row y: crop, GELU
template <typename IO>
__device__ __forceinline__ void store_crop(const Params& P, IO* op, int y, int c, float2 v) {
  const int oy = y - P.p;
  if ((unsigned)oy >= (unsigned)P.H) return;
  const int ox = 2 * c - P.p;
  float a = v.x, b = -v.y;
  if (P.gelu) gelu_pair(a, b);
  IO* o = op + (size_t)(oy * P.W + ox);
  if (P.vec) {    // p and W even: both columns are inside or outside, and aligned
    if ((unsigned)ox < (unsigned)P.W) {
      if constexpr (sizeof(IO) == 4) {
        *(float2*)o = make_float2(a, b);
      } else {
        *(__nv_bfloat162*)o = __floats2bfloat162_rn(a, b);
      }
    }
  } else {
    if ((unsigned)ox < (unsigned)P.W) st_io<IO>(o, 0, a);
    if ((unsigned)(ox + 1) < (unsigned)P.W) st_io<IO>(o, 1, b);
  }
}

// ------------------------------------------------------------------ columns forward: x -> S^
// CSH: log2 of the lines of a block, or -1 for the run-time value.  Shared memory: the tile [pos][line], then the row
// offsets.  Lanes run along the lines, so every access of a half warp is one contiguous piece of a row.
template <typename IO, int MAXR, int CSH>
__device__ __forceinline__ void cols_fwd_body(const Params& P, float2* T) {
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int sh = CSH >= 0 ? CSH : P.lsh_c, NL = 1 << sh;
  const int l = tid & (NL - 1);
  const int gl = blockIdx.x * NL + l;
  const bool valid = gl < P.nplane * P.wc;
  const int pl = valid ? gl / P.wc : 0, c = valid ? gl - pl * P.wc : 0;
  ColumnPair<IO> cp;
  cp.set(P, (const IO*)P.x + (size_t)(P.plane0 + pl) * P.H * P.W, c, valid);
  const Axis& ay = P.ay;
  const int r0 = ay.r0, r1 = ay.r1;
  float2* Tl = T + l;
  int* rowoff = (int*)(T + ((size_t)P.h << sh));
  for (int y = tid; y < P.h; y += nthr) rowoff[y] = row_offset(P, y);
  __syncthreads();
  if (MAXR <= kSmallRadix || ay.nkg == 0) {
    dispatch<MAXR>(r0, [&](auto ic) {
      constexpr int R = decltype(ic)::value;
      for (int j = tid >> sh; j < r1; j += nthr >> sh) {
        float re[R], im[R];
        load_rows<R, IO>(P, cp, rowoff, j, r1, re, im);
        Radix<R>::fwd(re, im);
#pragma unroll
        for (int k = 0; k < R; ++k) Tl[(k * r1 + j) << sh] = make_float2(re[k], im[k]);
      }
    });
  } else {
    for (int y0 = tid >> sh; y0 < P.h; y0 += 8 * (nthr >> sh)) {
      float re[8], im[8];
      const int step = nthr >> sh;
      if (y0 + 7 * step < P.h) {
        load_rows<8, IO>(P, cp, rowoff, y0, step, re, im);
#pragma unroll
        for (int u = 0; u < 8; ++u) Tl[(y0 + u * step) << sh] = make_float2(re[u], im[u]);
      } else {
        for (int y = y0; y < P.h; y += step) {
          float a[1], b[1];
          load_rows<1, IO>(P, cp, rowoff, y, 0, a, b);
          Tl[y << sh] = make_float2(a[0], b[0]);
        }
      }
    }
    __syncthreads();
    // vector v = (j, line): elements (j + r1 q, line) in, (k r1 + j, line) out -- the same set of cells
    matrix_stage<true>(ay, r1 << sh,
                       [&](int v, int q) { return T[v + ((r1 * q) << sh)]; },
                       [&](int v, int k, float2 z) { T[v + ((r1 * k) << sh)] = z; });
  }
  __syncthreads();
  // radix R1; lanes with bit `sh` clear hold k0 = kk, those with it set R0 - kk, so that Z[k] and Z[-k] are
  // one shuffle apart
  float2* wl = P.ws + ((size_t)pl * P.hh) * P.wp + 2 * c;
  dispatch<MAXR>(r1, [&](auto ic) {
    constexpr int R = decltype(ic)::value;
    constexpr int JH = (R + 1) / 2;
    const int per = nthr >> (sh + 1), side = (tid >> sh) & 1;
    for (int kb = 0; kb <= r0 / 2; kb += per) {
      const int kk = kb + (tid >> (sh + 1));
      const bool in = kk <= r0 / 2;
      if (!__any_sync(0xffffffffu, in)) break;
      const bool self = kk == 0 || 2 * kk == r0;
      const int k0 = !in || kk == 0 ? 0 : side ? r0 - kk : kk;
      float re[R], im[R];
      const float2* tp = Tl + ((k0 * r1) << sh);
#pragma unroll
      for (int j = 0; j < R; ++j) {
        const float2 v = tp[j << sh];
        re[j] = v.x; im[j] = v.y;
      }
      twiddle<R>(re, im, ay.tw + k0 * r1);
      Radix<R>::fwd(re, im);
      const bool st = in && valid && !(self && side);
      float2* wr = wl + (size_t)k0 * P.wp;
      const size_t ws = (size_t)r0 * P.wp;
      auto put = [&](int j2, float wx, float wy) {
        *(float4*)(wr + j2 * ws) = make_float4(re[j2] + wx, im[j2] - wy, im[j2] + wy, wx - re[j2]);
      };
      // all 16 lines of a warp share kk when a block has 16 lines: the branches are then warp-uniform
      if (CSH == 4 && self) {
        if (st) {
          if (kk == 0) {
#pragma unroll
            for (int j2 = 0; j2 <= R / 2; ++j2) put(j2, re[(R - j2) % R], im[(R - j2) % R]);
          } else {
#pragma unroll
            for (int j2 = 0; j2 < JH; ++j2) put(j2, re[R - 1 - j2], im[R - 1 - j2]);
          }
        }
      } else {
#pragma unroll
        for (int j2 = 0; j2 < JH; ++j2) {
          float wx = __shfl_xor_sync(0xffffffffu, re[R - 1 - j2], NL);
          float wy = __shfl_xor_sync(0xffffffffu, im[R - 1 - j2], NL);
          if (CSH != 4) {
            if (self) { wx = re[R - 1 - j2]; wy = im[R - 1 - j2]; }
            if (kk == 0) { wx = re[(R - j2) % R]; wy = im[(R - j2) % R]; }
          }
          if (st && !((R & 1) && j2 == JH - 1 && side)) put(j2, wx, wy);
        }
        if (CSH != 4 && (R & 1) == 0 && kk == 0 && st) put(R / 2, re[R / 2], im[R / 2]);
      }
    }
  });
}

// ------------------------------------------------------------------ rows: S^ -> . table -> U, in place
// R1-point butterfly of row `row` at k0, multiply, conjugate, R1-point butterfly, in place in shared memory
template <int R>
__device__ __forceinline__ void rows_mid(const Params& P, float2* Tk, const float2* tab, int k0) {
  const Axis& ax = P.ax;
  float re[R], im[R];
  const size_t ts = (size_t)ax.r0 * P.hh;
  const float2* tp = tab + (size_t)k0 * P.hh;
  const float2* tw = ax.tw + k0 * ax.r1;
  constexpr bool kAhead = R <= 10;       // table values requested before the butterfly while registers allow
  float2 g[R];
  if (kAhead) {
#pragma unroll
    for (int j2 = 0; j2 < R; ++j2) g[j2] = __ldg(tp + j2 * ts);
  }
#pragma unroll
  for (int j = 0; j < R; ++j) {
    const float2 v = Tk[j];
    re[j] = v.x; im[j] = v.y;
  }
  twiddle<R>(re, im, tw);
  Radix<R>::fwd(re, im);
  const float sg = P.conj ? -1.f : 1.f;
  if (!kAhead) {
#pragma unroll
    for (int j2 = 0; j2 < R; ++j2) g[j2] = __ldg(tp + j2 * ts);
  }
#pragma unroll
  for (int j2 = 0; j2 < R; ++j2) {
    const float xr = re[j2], xi = im[j2], gy = sg * g[j2].y;
    re[j2] = fmaf(-xi, gy, xr * g[j2].x);
    im[j2] = -fmaf(xr, gy, xi * g[j2].x);
  }
  Radix<R>::fwd(re, im);
  twiddle<R>(re, im, tw);
#pragma unroll
  for (int j = 0; j < R; ++j) Tk[j] = make_float2(re[j], im[j]);
}

template <int MAXR, int CSH>
__device__ __forceinline__ void rows_body(const Params& P, float2* T) {
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int sh = CSH >= 0 ? CSH : P.lsh_r, NL = 1 << sh, pitch = P.pitch;
  const Axis& ax = P.ax;
  const int r0 = ax.r0, r1 = ax.r1;
  const int row0 = blockIdx.x * NL, nrows = P.nplane * P.hh;
  const int nl = nrows - row0 < NL ? nrows - row0 : NL;
  float2* W = P.ws + (size_t)row0 * P.wp;
  const bool matrix = MAXR > kSmallRadix && ax.nkg != 0;
  if (!matrix) {
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
    // whole rows into shared memory, a warp per row
    for (int row = tid >> 5; row < nl; row += nthr >> 5) {
      const float2* src = W + (size_t)row * P.wp;
      for (int x0 = tid & 31; x0 < P.w; x0 += 32 * 8) {
        float2 v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (x0 + 32 * u < P.w) v[u] = src[x0 + 32 * u];
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (x0 + 32 * u < P.w) T[row * pitch + x0 + 32 * u] = v[u];
      }
    }
    __syncthreads();
    matrix_stage<true>(ax, r1 << sh,
                       [&](int v, int q) { return T[(v & (NL - 1)) * pitch + (v >> sh) + r1 * q]; },
                       [&](int v, int k, float2 z) { T[(v & (NL - 1)) * pitch + (v >> sh) + r1 * k] = z; });
  }
  __syncthreads();
  {
    const int row = tid & (NL - 1);
    if (row < nl) {
      const int g = row0 + row, pl = g / P.hh, k = g - pl * P.hh;
      const int c = (P.plane0 + pl) % P.C;
      const float2* tab = P.tab + (size_t)c * P.w * P.hh + k;
      dispatch<MAXR>(r1, [&](auto ic) {
        constexpr int R = decltype(ic)::value;
        for (int k0 = tid >> sh; k0 < r0; k0 += nthr >> sh) rows_mid<R>(P, T + row * pitch + k0 * r1, tab, k0);
      });
    }
  }
  __syncthreads();
  if (!matrix) {
    dispatch<MAXR>(r0, [&](auto ic) {
      constexpr int R = decltype(ic)::value;
      for (int it = tid; it < nl * r1; it += nthr) {
        int row, j;
        divmod_small(it, r1, ax.inv_r1, row, j);
        const float2* src = T + row * pitch + j;
        float re[R], im[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
          const float2 v = src[r1 * q];
          re[q] = v.x; im[q] = v.y;
        }
        Radix<R>::fwd(re, im);
        float2* dst = W + (size_t)row * P.wp + j;
#pragma unroll
        for (int k = 0; k < R; ++k) dst[k * r1] = make_float2(re[k], im[k]);
      }
    });
  } else {
    matrix_stage<true>(ax, r1 << sh,
                       [&](int v, int q) { return T[(v & (NL - 1)) * pitch + (v >> sh) + r1 * q]; },
                       [&](int v, int k, float2 z) { T[(v & (NL - 1)) * pitch + (v >> sh) + r1 * k] = z; });
    __syncthreads();
    for (int row = tid >> 5; row < nl; row += nthr >> 5) {
      float2* dst = W + (size_t)row * P.wp;
      for (int x = tid & 31; x < P.w; x += 32) dst[x] = T[row * pitch + x];
    }
  }
}

// ------------------------------------------------------------------ columns inverse: U -> out (or r)
template <typename IO, int MAXR, int CSH>
__device__ __forceinline__ void cols_inv_body(const Params& P, float2* T) {
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int sh = CSH >= 0 ? CSH : P.lsh_c, NL = 1 << sh;
  const int l = tid & (NL - 1);
  const int gl = blockIdx.x * NL + l;
  const bool valid = gl < P.nplane * P.wc;
  const int pl = valid ? gl / P.wc : 0, c = valid ? gl - pl * P.wc : 0;
  const Axis& ay = P.ay;
  const int r0 = ay.r0, r1 = ay.r1;
  float2* Tl = T + l;
  const float2* wl = P.ws + ((size_t)pl * P.hh) * P.wp + 2 * c;
  dispatch<MAXR>(r1, [&](auto ic) {
    constexpr int R = decltype(ic)::value;
    constexpr int JH = (R + 1) / 2;
    const int per = nthr >> (sh + 1), side = (tid >> sh) & 1;
    for (int kb = 0; kb <= r0 / 2; kb += per) {
      const int kk = kb + (tid >> (sh + 1));
      const bool in = kk <= r0 / 2;
      if (!__any_sync(0xffffffffu, in)) break;
      const bool self = kk == 0 || 2 * kk == r0;
      const int k0 = !in || kk == 0 ? 0 : side ? r0 - kk : kk;
      float re[R], im[R];
      const float2* wr = wl + (size_t)k0 * P.wp;
      const size_t ws = (size_t)r0 * P.wp;
      float4 u[JH];
#pragma unroll
      for (int j2 = 0; j2 < JH; ++j2) {
        // row k0 + r0 j2 <= h / 2, except the middle one of side 1 for odd R
        const bool have = !((R & 1) && j2 == JH - 1 && side && !self);
        u[j2] = have ? *(const float4*)(wr + j2 * ws) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
      // V[k] of a row's pair of columns, and V[h - k]
      auto v1x = [&](const float4& a) { return a.x + a.w; };
      auto v1y = [&](const float4& a) { return a.y - a.z; };
      auto v2x = [&](const float4& a) { return a.x - a.w; };
      auto v2y = [&](const float4& a) { return -a.y - a.z; };
#pragma unroll
      for (int j2 = 0; j2 < JH; ++j2) { re[j2] = v1x(u[j2]); im[j2] = v1y(u[j2]); }
      if (CSH == 4 && self) {            // warp-uniform: k0 = 0 or R0 / 2 is its own mirror
        if (kk == 0) {
          float4 uh = make_float4(0.f, 0.f, 0.f, 0.f);
          if ((R & 1) == 0) uh = *(const float4*)(wr + (R / 2) * ws);
#pragma unroll
          for (int j2 = 1; j2 < JH; ++j2) { re[R - j2] = v2x(u[j2]); im[R - j2] = v2y(u[j2]); }
          if ((R & 1) == 0) { re[R / 2] = v1x(uh); im[R / 2] = v1y(uh); }
        } else {
#pragma unroll
          for (int j2 = 0; j2 < R / 2; ++j2) { re[R - 1 - j2] = v2x(u[j2]); im[R - 1 - j2] = v2y(u[j2]); }
        }
      } else {
        float4 uh = make_float4(0.f, 0.f, 0.f, 0.f);
        if (CSH != 4 && (R & 1) == 0 && kk == 0) uh = *(const float4*)(wr + (R / 2) * ws);
#pragma unroll
        for (int j2 = 0; j2 < JH; ++j2) {
          const float ax_ = v2x(u[j2]), ay_ = v2y(u[j2]);
          float wx = __shfl_xor_sync(0xffffffffu, ax_, NL);
          float wy = __shfl_xor_sync(0xffffffffu, ay_, NL);
          if (R - 1 - j2 != j2) {
            if (CSH != 4) {
              const int n = j2 + 1 < JH ? j2 + 1 : j2;
              float ox = v2x(u[n]), oy = v2y(u[n]);
              if ((R & 1) == 0 && j2 == JH - 1) { ox = v1x(uh); oy = v1y(uh); }
              if (self) { wx = ax_; wy = ay_; }
              if (kk == 0) { wx = ox; wy = oy; }
            }
            re[R - 1 - j2] = wx; im[R - 1 - j2] = wy;
          } else if (side && !self) {
            re[j2] = wx; im[j2] = wy;
          }
        }
      }
      Radix<R>::fwd(re, im);
      twiddle<R>(re, im, ay.tw + k0 * r1);
      if (in && !(self && side)) {
        float2* tp = Tl + ((k0 * r1) << sh);
#pragma unroll
        for (int j = 0; j < R; ++j) tp[j << sh] = make_float2(re[j], im[j]);
      }
    }
  });
  __syncthreads();
  if (MAXR <= kSmallRadix || ay.nkg == 0) {
    if (!valid) return;
    IO* op = (IO*)P.out + (size_t)(P.plane0 + pl) * P.H * P.W;
    float2* rl = (float2*)P.r + (size_t)pl * P.h * P.wc + c;
    dispatch<MAXR>(r0, [&](auto ic) {
      constexpr int R = decltype(ic)::value;
      for (int j = tid >> sh; j < r1; j += nthr >> sh) {
        float re[R], im[R];
#pragma unroll
        for (int k = 0; k < R; ++k) {
          const float2 v = Tl[(k * r1 + j) << sh];
          re[k] = v.x; im[k] = v.y;
        }
        Radix<R>::fwd(re, im);
        if (P.s == 1) {
#pragma unroll
          for (int q = 0; q < R; ++q) store_crop<IO>(P, op, j + r1 * q, c, make_float2(re[q], im[q]));
        } else {
#pragma unroll
          for (int q = 0; q < R; ++q) rl[(size_t)(j + r1 * q) * P.wc] = make_float2(re[q], -im[q]);
        }
      }
    });
  } else {
    // the matrix stage's vectors are (j, line) with any line of the block: line data are recomputed per vector
    matrix_stage<false>(ay, r1 << sh,
                        [&](int v, int q) { return T[v + ((q * r1) << sh)]; },
                        [&](int v, int q, float2 z) {
                          const int g = blockIdx.x * NL + (v & (NL - 1));
                          if (g >= P.nplane * P.wc) return;
                          const int vp = g / P.wc, vcol = g - vp * P.wc, y = (v >> sh) + r1 * q;
                          if (P.s == 1)
                            store_crop<IO>(P, (IO*)P.out + (size_t)(P.plane0 + vp) * P.H * P.W, y, vcol, z);
                          else
                            ((float2*)P.r)[((size_t)vp * P.h + y) * P.wc + vcol] = make_float2(z.x, -z.y);
                        });
  }
}

// ------------------------------------------------------------------ upsampling epilogue of one plane
// out[i][j] = x[i/s][j/s] + sum_{a,b} K[a][b] Z[i+a-c][j+b-c], Z = zero_insert(r) on the circular
// s h x s w grid, cropped.  r: row-major reals, pitch `rp`.  A thread owns CW low-resolution columns and rows
// my0 .. my1 - 1 with a sliding window of r.
template <int S, int K, int CW, typename IO>
__device__ __forceinline__ void epi_rows(const Params& P, const float* r, int rp, const float* wk, const IO* xp, IO* op,
                                         int sx, int my0, int my1) {
  constexpr int c = K / 2;
  constexpr int DMIN = (c == 0) ? 0 : -((c + S - 1) / S);
  constexpr int DMAX = (S - 1 + K - 1 - c) / S;
  constexpr int WIN = DMAX - DMIN + 1, WC = CW + WIN - 1, NO = CW * S;
  const int h = P.h, w = P.w, p = P.p, oW = P.W * S;
  const int mx0 = sx * CW;
  const int ncell = P.W - mx0 < CW ? P.W - mx0 : CW;
  float kw[K * K];
#pragma unroll
  for (int i = 0; i < K * K; ++i) kw[i] = wk[i];
  int cols[WC];
#pragma unroll
  for (int e = 0; e < WC; ++e) {
    int n = mx0 + p + DMIN + e;
    if (n < 0) n += w;
    if (n >= w) n -= w;
    if (n >= w) n -= w;
    if (n < 0 || n >= w) n = 0;      // columns past a short last strip
    cols[e] = n;
  }
  const bool vec = ncell == CW && (oW * (int)sizeof(IO)) % 16 == 0 && (NO * (int)sizeof(IO)) % 16 == 0 &&
                   ((size_t)op) % 16 == 0;
  float win[WIN][WC];
  int rm = my0 + p + DMIN;
  if (rm < 0) rm += h;
  if (rm >= h) rm -= h;
#pragma unroll
  for (int d = 0; d + 1 < WIN; ++d) {
#pragma unroll
    for (int e = 0; e < WC; ++e) win[d][e] = r[(size_t)rm * rp + cols[e]];
    rm = rm + 1 == h ? 0 : rm + 1;
  }
  for (int my = my0; my < my1; ++my) {
#pragma unroll
    for (int e = 0; e < WC; ++e) win[WIN - 1][e] = r[(size_t)rm * rp + cols[e]];
    rm = rm + 1 == h ? 0 : rm + 1;
    float ya[CW];
#pragma unroll
    for (int e = 0; e < CW; ++e) ya[e] = ld_io<IO>(xp, (size_t)(my * P.W + mx0 + (e < ncell ? e : 0)));
#pragma unroll
    for (int da = 0; da < S; ++da) {
      float oa[NO];
#pragma unroll
      for (int e = 0; e < CW; ++e) {
#pragma unroll
        for (int db = 0; db < S; ++db) {
          float acc = ya[e];
#pragma unroll
          for (int a = 0; a < K; ++a) {
            const int ii = da + a - c;
            const int fi = (ii >= 0) ? ii / S : -((-ii + S - 1) / S);
            if (ii - fi * S != 0) continue;
#pragma unroll
            for (int b = 0; b < K; ++b) {
              const int jj = db + b - c;
              const int fj = (jj >= 0) ? jj / S : -((-jj + S - 1) / S);
              if (jj - fj * S != 0) continue;
              acc = fmaf(kw[a * K + b], win[fi - DMIN][e + fj - DMIN], acc);
            }
          }
          oa[e * S + db] = acc;
        }
      }
      if (P.gelu) {
#pragma unroll
        for (int i = 0; i < NO; i += 2) {
          if (i + 1 < NO) gelu_pair(oa[i], oa[i + 1]);
          else oa[i] = gelu_erf(oa[i]);
        }
      }
      IO* o = op + (size_t)(my * S + da) * oW + mx0 * S;
      if (vec) {
        if constexpr ((NO * sizeof(IO)) % 16 == 0) {
          if constexpr (sizeof(IO) == 4) {
#pragma unroll
            for (int i = 0; i < NO; i += 4) __stcs((float4*)(o + i), make_float4(oa[i], oa[i + 1], oa[i + 2], oa[i + 3]));
          } else {
#pragma unroll
            for (int i = 0; i < NO; i += 8) {
              __nv_bfloat162 v0 = __floats2bfloat162_rn(oa[i], oa[i + 1]), v1 = __floats2bfloat162_rn(oa[i + 2], oa[i + 3]);
              __nv_bfloat162 v2 = __floats2bfloat162_rn(oa[i + 4], oa[i + 5]), v3 = __floats2bfloat162_rn(oa[i + 6], oa[i + 7]);
              uint4 q;
              q.x = *(unsigned*)&v0; q.y = *(unsigned*)&v1; q.z = *(unsigned*)&v2; q.w = *(unsigned*)&v3;
              *(uint4*)(o + i) = q;
            }
          }
        }
      } else {
#pragma unroll
        for (int i = 0; i < NO; ++i)
          if (i < ncell * S) st_io<IO>(o, (size_t)i, oa[i]);
      }
    }
#pragma unroll
    for (int d = 0; d + 1 < WIN; ++d) {
#pragma unroll
      for (int e = 0; e < WC; ++e) win[d][e] = win[d + 1][e];
    }
  }
}

// any scale and tap count: one low-resolution cell
template <typename IO>
__device__ __forceinline__ void epi_cell(const Params& P, const float* r, int rp, const float* wk, const IO* xp, IO* op,
                                         int my, int mx) {
  const int s = P.s, k = P.k, cc = P.k / 2, h = P.h, w = P.w, oW = P.W * s;
  const float y = ld_io<IO>(xp, (size_t)(my * P.W + mx));
  for (int da = 0; da < s; ++da)
    for (int db = 0; db < s; ++db) {
      float acc = y;
      const int a0 = ((cc - da) % s + s) % s, b0 = ((cc - db) % s + s) % s;   // first tap whose offset is a multiple of s
      for (int a = a0; a < k; a += s) {
        int rm = (my + P.p + (da + a - cc) / s) % h;
        if (rm < 0) rm += h;
        for (int b = b0; b < k; b += s) {
          int rn = (mx + P.p + (db + b - cc) / s) % w;
          if (rn < 0) rn += w;
          acc = fmaf(wk[a * k + b], r[(size_t)rm * rp + rn], acc);
        }
      }
      st_io<IO>(op, (size_t)(my * s + da) * oW + (size_t)(mx * s + db), P.gelu ? gelu_erf(acc) : acc);
    }
}

#define CVB_RP_EPI_CASES(X) X(2, 2, 2, 4) X(2, 3, 2, 4) X(2, 5, 2, 4) X(2, 7, 2, 4) X(3, 3, 4, 4) X(3, 5, 4, 4) X(3, 7, 4, 4) X(4, 3, 1, 2) X(4, 5, 1, 2) X(4, 7, 1, 2)

// rows my0 .. my0 + nr - 1 (clipped) of strips sx0, sx0 + step, ...; `items` threads cooperate with index `t`
template <typename IO>
__device__ __forceinline__ void epilogue(const Params& P, const float* r, int rp, const float* wk, const IO* xp, IO* op,
                                         int t, int items, int my0, int my1) {
  const int key = P.s * 16 + P.k;
  switch (key) {
#define X(S_, K_, CWF, CWB)                                                                             \
  case S_ * 16 + K_: {                                                                                  \
    constexpr int CW = sizeof(IO) == 4 ? CWF : CWB;                                                     \
    const int spr = (P.W + CW - 1) / CW;                                                                \
    int nseg = items / spr;                                                                             \
    const int rows = my1 - my0;                                                                         \
    if (nseg < 1) nseg = 1;                                                                             \
    if (nseg > rows) nseg = rows;                                                                       \
    const int rps = (rows + nseg - 1) / nseg;                                                           \
    for (int i = t; i < spr * nseg; i += items) {                                                       \
      const int seg = i / spr, sx = i - seg * spr;                                                      \
      const int b0 = my0 + seg * rps, b1 = b0 + rps < my1 ? b0 + rps : my1;                             \
      if (b0 < b1) epi_rows<S_, K_, CW, IO>(P, r, rp, wk, xp, op, sx, b0, b1);                          \
    }                                                                                                   \
  } break;
    CVB_RP_EPI_CASES(X)
#undef X
    default:
      for (int i = t; i < (my1 - my0) * P.W; i += items) {
        const int my = my0 + i / P.W, mx = i % P.W;
        epi_cell<IO>(P, r, rp, wk, xp, op, my, mx);
      }
  }
}

// ------------------------------------------------------------------ one plane per block, all in shared memory
// T1[pos][c] (h x wc, then r), T2[k][x] (hh rows of odd pitch), the taps, the row offsets.
template <typename IO, int MAXR>
__device__ __forceinline__ void plane_body(const Params& P, float2* sm) {
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int h = P.h, w = P.w, hh = P.hh, wc = P.wc, pitch = P.pitch;
  float2* T1 = sm;
  float2* T2 = sm + (size_t)h * wc;
  float* wk = (float*)(T2 + (size_t)hh * pitch);
  int* rowoff = (int*)(wk + ((P.k * P.k + 1) & ~1));
  const int plane = P.plane0 + blockIdx.x, ch = plane % P.C;
  const IO* xp = (const IO*)P.x + (size_t)plane * P.H * P.W;
  const Axis& ay = P.ay;
  const Axis& ax = P.ax;
  const bool my_ = MAXR > kSmallRadix && ay.nkg != 0, mx_ = MAXR > kSmallRadix && ax.nkg != 0;
  if (P.s > 1)
    for (int i = tid; i < P.k * P.k; i += nthr) wk[i] = P.weight[(size_t)ch * P.k * P.k + i];
  for (int y = tid; y < h; y += nthr) rowoff[y] = row_offset(P, y);
  __syncthreads();
  // ---- columns forward
  {
    const int r0 = ay.r0, r1 = ay.r1, st = r1 * wc;
    if (!my_) {
      dispatch<MAXR>(r0, [&](auto ic) {
        constexpr int R = decltype(ic)::value;
        for (int it = tid; it < st; it += nthr) {
          int j, c;
          divmod_small(it, wc, P.inv_wc, j, c);
          ColumnPair<IO> cp;
          cp.set(P, xp, c, true);
          float re[R], im[R];
          load_rows<R, IO>(P, cp, rowoff, j, r1, re, im);
          Radix<R>::fwd(re, im);
          float2* d = T1 + it;
#pragma unroll
          for (int k = 0; k < R; ++k) d[k * st] = make_float2(re[k], im[k]);
        }
      });
    } else {
      for (int it = tid; it < h * wc; it += nthr) {
        int y, c;
        divmod_small(it, wc, P.inv_wc, y, c);
        ColumnPair<IO> cp;
        cp.set(P, xp, c, true);
        float re[1], im[1];
        load_rows<1, IO>(P, cp, rowoff, y, 0, re, im);
        T1[it] = make_float2(re[0], im[0]);
      }
      __syncthreads();
      matrix_stage<true>(ay, st, [&](int v, int q) { return T1[v + q * st]; },
                         [&](int v, int k, float2 z) { T1[v + k * st] = z; });
    }
    __syncthreads();
    // radix R1 of k0 = kk and of its mirror R0 - kk in one thread, spectra of the two columns separated
    const int nkk = r0 / 2 + 1;
    dispatch<MAXR>(r1, [&](auto ic) {
      constexpr int R = decltype(ic)::value;
      constexpr int JH = (R + 1) / 2;
      for (int it = tid; it < nkk * wc; it += nthr) {
        int kk, c;
        divmod_small(it, wc, P.inv_wc, kk, c);
        const bool two = 2 * c + 1 < w;
        float2* out = T2 + 2 * c;
        auto put = [&](int k, float zr, float zi, float wr, float wi) {
          float2* o = out + k * pitch;
          o[0] = make_float2(zr + wr, zi - wi);
          if (two) o[1] = make_float2(zi + wi, wr - zr);
        };
        float ar[R], ai[R];
        const float2* s0 = T1 + kk * st + c;
#pragma unroll
        for (int j = 0; j < R; ++j) {
          const float2 v = s0[j * wc];
          ar[j] = v.x; ai[j] = v.y;
        }
        twiddle<R>(ar, ai, ay.tw + kk * r1);
        Radix<R>::fwd(ar, ai);
        if (kk == 0) {
#pragma unroll
          for (int j2 = 0; j2 <= R / 2; ++j2) put(r0 * j2, ar[j2], ai[j2], ar[(R - j2) % R], ai[(R - j2) % R]);
        } else if (2 * kk == r0) {
#pragma unroll
          for (int j2 = 0; j2 < JH; ++j2) put(kk + r0 * j2, ar[j2], ai[j2], ar[R - 1 - j2], ai[R - 1 - j2]);
        } else {
          float br[R], bi[R];
          const float2* s1 = T1 + (r0 - kk) * st + c;
#pragma unroll
          for (int j = 0; j < R; ++j) {
            const float2 v = s1[j * wc];
            br[j] = v.x; bi[j] = v.y;
          }
          twiddle<R>(br, bi, ay.tw + (r0 - kk) * r1);
          Radix<R>::fwd(br, bi);
#pragma unroll
          for (int j2 = 0; j2 < JH; ++j2) put(kk + r0 * j2, ar[j2], ai[j2], br[R - 1 - j2], bi[R - 1 - j2]);
#pragma unroll
          for (int j2 = 0; j2 < R / 2; ++j2) put(r0 - kk + r0 * j2, br[j2], bi[j2], ar[R - 1 - j2], ai[R - 1 - j2]);
        }
      }
    });
    __syncthreads();
  }
  // ---- rows, in place in T2
  {
    const int r0 = ax.r0, r1 = ax.r1;
    const float2* tab = P.tab + (size_t)ch * w * hh;
    auto outer = [&]() {
      if (!mx_) {
        dispatch<MAXR>(r0, [&](auto ic) {
          constexpr int R = decltype(ic)::value;
          for (int it = tid; it < hh * r1; it += nthr) {
            int row, j;
            divmod_small(it, r1, ax.inv_r1, row, j);
            float2* d = T2 + row * pitch + j;
            float re[R], im[R];
#pragma unroll
            for (int q = 0; q < R; ++q) {
              const float2 v = d[q * r1];
              re[q] = v.x; im[q] = v.y;
            }
            Radix<R>::fwd(re, im);
#pragma unroll
            for (int k = 0; k < R; ++k) d[k * r1] = make_float2(re[k], im[k]);
          }
        });
      } else {
        matrix_stage<true>(ax, r1 * hh,
                           [&](int v, int q) { int j, row; divmod_small(v, hh, P.inv_hh, j, row); return T2[row * pitch + j + r1 * q]; },
                           [&](int v, int k, float2 z) { int j, row; divmod_small(v, hh, P.inv_hh, j, row); T2[row * pitch + j + r1 * k] = z; });
      }
      __syncthreads();
    };
    // the two outer passes share one copy of the butterfly code
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
      outer();
      if (pass == 0) {
        dispatch<MAXR>(r1, [&](auto ic) {
          constexpr int R = decltype(ic)::value;
          for (int it = tid; it < r0 * hh; it += nthr) {
            int k0, row;
            divmod_small(it, hh, P.inv_hh, k0, row);
            rows_mid<R>(P, T2 + row * pitch + k0 * r1, tab + row, k0);
          }
        });
        __syncthreads();
      }
    }
  }
  // ---- columns inverse
  {
    const int r0 = ay.r0, r1 = ay.r1, st = r1 * wc, nkk = r0 / 2 + 1;
    dispatch<MAXR>(r1, [&](auto ic) {
      constexpr int R = decltype(ic)::value;
      constexpr int JH = (R + 1) / 2;
      for (int it = tid; it < nkk * wc; it += nthr) {
        int kk, c;
        divmod_small(it, wc, P.inv_wc, kk, c);
        const bool two = 2 * c + 1 < w;
        const float2* in = T2 + 2 * c;
        auto get = [&](int k, float2& e, float2& o) {
          e = in[k * pitch];
          o = two ? in[k * pitch + 1] : make_float2(0.f, 0.f);
        };
        auto finish = [&](float (&re)[R], float (&im)[R], int k0) {
          Radix<R>::fwd(re, im);
          twiddle<R>(re, im, ay.tw + k0 * r1);
          float2* d = T1 + k0 * st + c;
#pragma unroll
          for (int j = 0; j < R; ++j) d[j * wc] = make_float2(re[j], im[j]);
        };
        float ar[R], ai[R];
        float2 e, o;
        if (kk == 0) {
#pragma unroll
          for (int j2 = 0; j2 <= R / 2; ++j2) {
            get(r0 * j2, e, o);
            ar[j2] = e.x + o.y; ai[j2] = e.y - o.x;
            if (j2 > 0 && R - j2 != j2) { ar[(R - j2) % R] = e.x - o.y; ai[(R - j2) % R] = -e.y - o.x; }
          }
        } else if (2 * kk == r0) {
#pragma unroll
          for (int j2 = 0; j2 < JH; ++j2) {
            get(kk + r0 * j2, e, o);
            ar[j2] = e.x + o.y; ai[j2] = e.y - o.x;
            if (R - 1 - j2 != j2) { ar[R - 1 - j2] = e.x - o.y; ai[R - 1 - j2] = -e.y - o.x; }
          }
        } else {
          float br[R], bi[R];
#pragma unroll
          for (int j2 = 0; j2 < JH; ++j2) {
            get(kk + r0 * j2, e, o);
            ar[j2] = e.x + o.y; ai[j2] = e.y - o.x;
            br[R - 1 - j2] = e.x - o.y; bi[R - 1 - j2] = -e.y - o.x;
          }
#pragma unroll
          for (int j2 = 0; j2 < R / 2; ++j2) {
            get(r0 - kk + r0 * j2, e, o);
            br[j2] = e.x + o.y; bi[j2] = e.y - o.x;
            ar[R - 1 - j2] = e.x - o.y; ai[R - 1 - j2] = -e.y - o.x;
          }
          finish(br, bi, r0 - kk);
        }
        finish(ar, ai, kk);
      }
    });
    __syncthreads();
    IO* op = (IO*)P.out + (size_t)plane * P.H * P.W * P.s * P.s;
    if (!my_) {
      dispatch<MAXR>(r0, [&](auto ic) {
        constexpr int R = decltype(ic)::value;
        for (int it = tid; it < st; it += nthr) {
          int j, c;
          divmod_small(it, wc, P.inv_wc, j, c);
          float2* d = T1 + it;
          float re[R], im[R];
#pragma unroll
          for (int k = 0; k < R; ++k) {
            const float2 v = d[k * st];
            re[k] = v.x; im[k] = v.y;
          }
          Radix<R>::fwd(re, im);
          if (P.s == 1) {
#pragma unroll
            for (int q = 0; q < R; ++q) store_crop<IO>(P, op, j + r1 * q, c, make_float2(re[q], im[q]));
          } else {
#pragma unroll
            for (int q = 0; q < R; ++q) d[q * st] = make_float2(re[q], -im[q]);
          }
        }
      });
    } else if (P.s == 1) {
      matrix_stage<false>(ay, st, [&](int v, int q) { return T1[v + q * st]; },
                          [&](int v, int q, float2 z) {
                            int j, c;
                            divmod_small(v, wc, P.inv_wc, j, c);
                            store_crop<IO>(P, op, j + r1 * q, c, z);
                          });
    } else {
      matrix_stage<true>(ay, st, [&](int v, int q) { return T1[v + q * st]; },
                         [&](int v, int q, float2 z) { T1[v + q * st] = make_float2(z.x, -z.y); });
    }
    if (P.s > 1) {
      __syncthreads();
      epilogue<IO>(P, (const float*)T1, 2 * wc, wk, xp, op, tid, nthr, 0, P.H);
    }
  }
}

// upsampling epilogue of the multi-launch form: grid (row segments, planes)
constexpr int kEpiRows = 16;
template <typename IO>
__device__ __forceinline__ void epilogue_body(const Params& P) {
  const int pl = blockIdx.y, plane = P.plane0 + pl, ch = plane % P.C;
  const int my0 = blockIdx.x * kEpiRows, my1 = my0 + kEpiRows < P.H ? my0 + kEpiRows : P.H;
  epilogue<IO>(P, P.r + (size_t)pl * P.h * P.wp, P.wp, P.weight + (size_t)ch * P.k * P.k,
               (const IO*)P.x + (size_t)plane * P.H * P.W, (IO*)P.out + (size_t)plane * P.H * P.W * P.s * P.s,
               threadIdx.x, blockDim.x, my0, my1);
}

}  // namespace rp
}  // namespace cvb
