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
  int mp;               // 0: R0 is a register butterfly; else the width of the matrix stage's rows
  float inv_r1;
  const float2* tw;     // twiddles in position order: [k0 r1 + j] = (cos, sin)(2 pi k0 j / n)
  const float* dm;      // matrix stage: cos(2 pi q k / R0) as [k = 0 .. R0/2][q = 1 .. mp], then sin likewise
  const unsigned char* fix;   // operand of the integer contractions (cvb_fix.cuh), or null
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
  int po, OH, OW;       // the output is the solved plane cropped to rows po .. po + OH - 1, columns likewise
  int vec, vec_out;     // pairs of columns are loaded (stored) at once: offset and width even, pointer aligned
  float2* ws;           // [nplane][hh][wp]
  float* r;             // scale >= 2: [nplane][h][wp]
  float* rsave;         // scale >= 2: all planes' r kept for the backward ([B C][h][wp]), or null
  int pitch;            // rows kernel / plane kernel: odd row pitch (complex) of the shared-memory rows
  float inv_wc, inv_hh;
  int* status;          // device word set non-zero when a bounded wait gives up; may be null
  Axis ay, ax;
};

__host__ __device__ constexpr bool register_radix(int r) {
#define CVB_RP_X(R) r == R ||
  return CVB_RP_EACH_RADIX(CVB_RP_X) false;
#undef CVB_RP_X
}
// Widths the matrix stage is built for (pairs q, R - q held in registers), and the one R0 takes: 0 = a register butterfly
#define CVB_RP_EACH_WIDTH(X) X(20) X(24) X(32) X(36) X(44) X(56) X(64)
__host__ __device__ constexpr int matrix_width(int r0) {
  if (register_radix(r0)) return 0;
#define CVB_RP_X(M) if (r0 / 2 <= M) return M;
  CVB_RP_EACH_WIDTH(CVB_RP_X)
#undef CVB_RP_X
  return -1;
}

// The smallest R0 / 2 that width M serves
__host__ __device__ constexpr int matrix_least(int m) {
  int least = 1;
#define CVB_RP_X(M) if (M < m) least = M + 1;
  CVB_RP_EACH_WIDTH(CVB_RP_X)
#undef CVB_RP_X
  return least;
}

// Builds of every kernel: both radices up to kSmallRadix (80 registers a thread); up to kAnyRadix; a matrix stage of a
// given width with R1 up to kMatrixR1.
constexpr int kSmallRadix = 20, kAnyRadix = 32, kMatrixR1 = 16;

constexpr int kLinesLog2 = 4, kLines = 16;   // lines (column pairs, rows) of a block of the strip kernels

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
// R-point transforms of nvec vectors in shared memory, in place; vector v has its elements at base(v)[q * stride].
// With p_q = x_q + x_(R-q), m_q = x_q - x_(R-q):  X_k = a_k - i b_k, X_(R-k) = a_k + i b_k,
// a_k = x_0 + sum_q cos(2 pi q k / R) p_q,  b_k = sum_q sin(2 pi q k / R) m_q.  One thread keeps the p (or the m) of a
// vector in registers and runs over the k: two FMAs per (k, q), the cosines four at a time from shared memory.  Element
// k then holds a_k and element R - k holds b_k (matrix_value puts them together), so that the two threads of a vector
// never have to meet.  About R FMAs per point; a 16-byte read of cosines (four cycles of the shared-memory port a warp)
// feeds eight of them a thread (two cycles of the FMA pipes), so the port is the nearer limit of the two.  Neither is
// reached: 1 x 128 planes of 268 x 268 keep the port below half busy, the FMA pipes a third and the issue slots a half, at
// 15 warps an SM (128 registers), waiting for memory.
template <int MP, class Base>
__device__ __forceinline__ void matrix_stage(int R, int nvec, int stride, const float* mats, Base base) {
  const int tid = threadIdx.x, half = blockDim.x >> 1;
  int nvr = (nvec + 15) & ~15;
  if (nvr > half) nvr = half;
  const int ng = half / nvr;                       // groups of k, when there are few vectors
  const int g = tid / nvr, vl = tid - g * nvr, side = g & 1, kg = g >> 1;
  const int KH = R >> 1, QH = (R - 1) >> 1;
  const int kper = (KH + ng) / ng;                 // rows k = 0 .. KH over the groups
  const float* mat = mats + (side ? (KH + 1) * MP : 0);
  for (int v0 = 0; v0 < nvec; v0 += nvr) {
    const bool act = v0 + vl < nvec && kg < ng;
    float2* x = base(act ? v0 + vl : 0);
    float2 p[MP];
    const float2 x0 = side ? make_float2(0.f, 0.f) : x[0];
    const float sg = side ? -1.f : 1.f;
    const float2 *up = x + stride, *dn = x + (R - 1) * stride;
#pragma unroll
    for (int q = 1; q <= MP; ++q, up += stride, dn -= stride) {
      if (q < matrix_least(MP) || q <= QH) {
        const float2 u = *up, w = *dn;
        p[q - 1] = make_float2(fmaf(sg, w.x, u.x), fmaf(sg, w.y, u.y));
      } else {
        p[q - 1] = make_float2(0.f, 0.f);
        if (q == KH && !side) p[q - 1] = *up;      // even R: the middle element, cosines only
      }
    }
    __syncthreads();
    if (act) {
      const int k0 = kg * kper > side ? kg * kper : side, k1 = (kg + 1) * kper < KH + 1 ? (kg + 1) * kper : KH + 1;
      const int kend = side && k1 > QH + 1 ? QH + 1 : k1;
      // two rows at a time: four independent sums, and one row's cosines arrive while the other's are used
      float2* o = x + (side ? R - k0 : k0) * stride;
      const int ostep = side ? -stride : stride;
#pragma unroll 1
      for (int k = k0; k < kend; k += 2, o += 2 * ostep) {
        const bool two = k + 1 < kend;
        const float4* c4 = (const float4*)(mat + k * MP);
        const float4* d4 = two ? c4 + MP / 4 : c4;
        float r0 = x0.x, i0 = x0.y, r1 = x0.x, i1 = x0.y;
#pragma unroll
        for (int q = 0; q < MP; q += 4) {
          const float4 c = c4[q >> 2], d = d4[q >> 2];
          r0 = fmaf(c.x, p[q].x, r0);     i0 = fmaf(c.x, p[q].y, i0);
          r1 = fmaf(d.x, p[q].x, r1);     i1 = fmaf(d.x, p[q].y, i1);
          r0 = fmaf(c.y, p[q + 1].x, r0); i0 = fmaf(c.y, p[q + 1].y, i0);
          r1 = fmaf(d.y, p[q + 1].x, r1); i1 = fmaf(d.y, p[q + 1].y, i1);
          r0 = fmaf(c.z, p[q + 2].x, r0); i0 = fmaf(c.z, p[q + 2].y, i0);
          r1 = fmaf(d.z, p[q + 2].x, r1); i1 = fmaf(d.z, p[q + 2].y, i1);
          r0 = fmaf(c.w, p[q + 3].x, r0); i0 = fmaf(c.w, p[q + 3].y, i0);
          r1 = fmaf(d.w, p[q + 3].x, r1); i1 = fmaf(d.w, p[q + 3].y, i1);
        }
        o[0] = make_float2(r0, i0);
        if (two) o[ostep] = make_float2(r1, i1);
      }
    }
  }
}
// element k of the transform from what matrix_stage leaves
__device__ __forceinline__ float2 matrix_value(const float2* x, int R, int k, int stride) {
  if (k == 0 || 2 * k == R) return x[k * stride];
  const bool mir = 2 * k > R;
  const float2 a = x[(mir ? R - k : k) * stride], b = x[(mir ? k : R - k) * stride];
  return mir ? make_float2(a.x - b.y, a.y + b.x) : make_float2(a.x + b.y, a.y - b.x);
}
// the R elements j = 0 .. R-1 of position kk (side 0) or r0 - kk (side 1), elements j at x + (j << sh)
template <int R>
__device__ __forceinline__ void load_matrix(const float2* x, int r0, int kk, int side, int stride, int sh, bool in,
                                            float (&re)[R], float (&im)[R]) {
  if (!in || kk == 0 || 2 * kk == r0) {
    const float2* a = x + (in ? kk : 0) * stride;
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const float2 v = a[j << sh];
      re[j] = v.x; im[j] = v.y;
    }
  } else {
    const float2* a = x + kk * stride;
    const float2* b = x + (r0 - kk) * stride;
    const float sg = side ? -1.f : 1.f;
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const float2 u = a[j << sh], v = b[j << sh];
      re[j] = fmaf(sg, v.y, u.x); im[j] = fmaf(-sg, v.x, u.y);
    }
  }
}
template <int MP>
__device__ __forceinline__ void copy_matrices(float* dst, const Axis& a) {
  const int n = 2 * (a.r0 / 2 + 1) * MP / 4;
  for (int i = threadIdx.x; i < n; i += blockDim.x) ((float4*)dst)[i] = __ldg((const float4*)a.dm + i);
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
  const int oy = y - P.po;
  if ((unsigned)oy >= (unsigned)P.OH) return;
  const int ox = 2 * c - P.po;
  float a = v.x, b = -v.y;
  if (P.gelu) gelu_fast_pair(a, b);
  IO* o = op + (size_t)(oy * P.OW + ox);
  if (P.vec_out) {    // both columns are inside or outside, and aligned
    if ((unsigned)ox < (unsigned)P.OW) {
      if constexpr (sizeof(IO) == 4) {
        *(float2*)o = make_float2(a, b);
      } else {
        *(__nv_bfloat162*)o = __floats2bfloat162_rn(a, b);
      }
    }
  } else {
    if ((unsigned)ox < (unsigned)P.OW) st_io<IO>(o, 0, a);
    if ((unsigned)(ox + 1) < (unsigned)P.OW) st_io<IO>(o, 1, b);
  }
}

// ------------------------------------------------------------------ columns forward: x -> S^
// A block takes 16 lines.  Shared memory: the tile [pos][line], then the row offsets.  Lanes run along the lines, so
// every access of a half warp is one contiguous piece of a row.
// MP > 0: the R0 points are a matrix stage of that width; its matrices follow the row offsets.
template <typename IO, int MAXR, int MP>
__device__ __forceinline__ void cols_fwd_body(const Params& P, float2* T) {
  const int tid = threadIdx.x, nthr = blockDim.x;
  constexpr int sh = kLinesLog2, NL = kLines;
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
  float* mats = (float*)(rowoff + ((P.h + 3) & ~3));
  if constexpr (MP > 0) copy_matrices<MP>(mats, ay);
  __syncthreads();
  if constexpr (MP == 0) {
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
    // vector v = (j, line): elements (j + r1 q, line) become (k r1 + j, line), the same cells
    matrix_stage<MP>(r0, r1 << sh, r1 << sh, mats, [&](int v) { return T + v; });
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
      if constexpr (MP == 0) {
#pragma unroll
        for (int j = 0; j < R; ++j) {
          const float2 v = tp[j << sh];
          re[j] = v.x; im[j] = v.y;
        }
      } else {
        load_matrix<R>(Tl, r0, kk, side, r1 << sh, sh, in, re, im);
      }
      twiddle<R>(re, im, ay.tw + k0 * r1);
      Radix<R>::fwd(re, im);
      const bool st = in && valid && !(self && side);
      float2* wr = wl + (size_t)k0 * P.wp;
      const size_t ws = (size_t)r0 * P.wp;
      auto put = [&](int j2, float wx, float wy) {
        *(float4*)(wr + j2 * ws) = make_float4(re[j2] + wx, im[j2] - wy, im[j2] + wy, wx - re[j2]);
      };
      if (self) {        // warp-uniform: a warp is 16 lines x 2 sides of one kk

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
          const float wx = __shfl_xor_sync(0xffffffffu, re[R - 1 - j2], NL);
          const float wy = __shfl_xor_sync(0xffffffffu, im[R - 1 - j2], NL);
          if (st && !((R & 1) && j2 == JH - 1 && side)) put(j2, wx, wy);
        }
      }
    }
  });
}

// ------------------------------------------------------------------ rows: S^ -> . table -> U, in place
// R1-point butterfly of a row at k0, multiply, conjugate, R1-point butterfly, to shared memory
template <int R>
__device__ __forceinline__ void rows_mid(const Params& P, float (&re)[R], float (&im)[R], float2* Tk, const float2* tab,
                                         int k0) {
  const Axis& ax = P.ax;
  const size_t ts = (size_t)ax.r0 * P.hh;
  const float2* tp = tab + (size_t)k0 * P.hh;
  const float2* tw = ax.tw + k0 * ax.r1;
  constexpr bool kAhead = R <= 10;       // table values requested before the butterfly while registers allow
  float2 g[R];
  if (kAhead) {
#pragma unroll
    for (int j2 = 0; j2 < R; ++j2) g[j2] = __ldg(tp + j2 * ts);
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

template <int MAXR, int MP>
__device__ __forceinline__ void rows_body(const Params& P, float2* T) {
  const int tid = threadIdx.x, nthr = blockDim.x;
  constexpr int sh = kLinesLog2, NL = kLines;
  const int pitch = P.pitch;
  const Axis& ax = P.ax;
  const int r0 = ax.r0, r1 = ax.r1;
  const int row0 = blockIdx.x * NL, nrows = P.nplane * P.hh;
  const int nl = nrows - row0 < NL ? nrows - row0 : NL;
  float2* W = P.ws + (size_t)row0 * P.wp;
  float* mats = (float*)(T + (((size_t)pitch << sh) + 1 & ~(size_t)1));
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
    copy_matrices<MP>(mats, ax);
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
    matrix_stage<MP>(r0, r1 << sh, r1, mats, [&](int v) { return T + (v & (NL - 1)) * pitch + (v >> sh); });
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
        if constexpr (MP == 0) {
          for (int k0 = tid >> sh; k0 < r0; k0 += nthr >> sh) {
            float2* Tk = T + row * pitch + k0 * r1;
            float re[R], im[R];
#pragma unroll
            for (int j = 0; j < R; ++j) {
              const float2 v = Tk[j];
              re[j] = v.x; im[j] = v.y;
            }
            rows_mid<R>(P, re, im, Tk, tab, k0);
          }
        } else {
          // positions kk and r0 - kk share what they read: one thread takes both
          float2* Tr = T + row * pitch;
          for (int kk = tid >> sh; kk <= r0 / 2; kk += nthr >> sh) {
            const bool self = kk == 0 || 2 * kk == r0;
            float ar[R], ai[R], br[R], bi[R];
#pragma unroll
            for (int j = 0; j < R; ++j) {
              const float2 u = Tr[kk * r1 + j], v = self ? make_float2(0.f, 0.f) : Tr[(r0 - kk) * r1 + j];
              ar[j] = u.x; ai[j] = u.y; br[j] = v.x; bi[j] = v.y;
            }
#pragma unroll 1
            for (int side = 0; side < (self ? 1 : 2); ++side) {
              const float sg = side ? -1.f : 1.f;
              const int k0 = side ? r0 - kk : kk;
              float re[R], im[R];
#pragma unroll
              for (int j = 0; j < R; ++j) { re[j] = fmaf(sg, bi[j], ar[j]); im[j] = fmaf(-sg, br[j], ai[j]); }
              rows_mid<R>(P, re, im, Tr + k0 * r1, tab, k0);
            }
          }
        }
      });
    }
  }
  __syncthreads();
  if constexpr (MP == 0) {
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
    matrix_stage<MP>(r0, r1 << sh, r1, mats, [&](int v) { return T + (v & (NL - 1)) * pitch + (v >> sh); });
    __syncthreads();
    for (int row = tid >> 5; row < nl; row += nthr >> 5) {
      float2* dst = W + (size_t)row * P.wp;
      for (int x = tid & 31; x < P.w; x += 32) {
        int q, j;
        divmod_small(x, r1, ax.inv_r1, q, j);
        dst[x] = matrix_value(T + row * pitch + j, r0, q, r1);
      }
    }
  }
}

// ------------------------------------------------------------------ columns inverse: U -> out (or r)
template <typename IO, int MAXR, int MP>
__device__ __forceinline__ void cols_inv_body(const Params& P, float2* T) {
  const int tid = threadIdx.x, nthr = blockDim.x;
  constexpr int sh = kLinesLog2, NL = kLines;
  const int l = tid & (NL - 1);
  const int gl = blockIdx.x * NL + l;
  const bool valid = gl < P.nplane * P.wc;
  const int pl = valid ? gl / P.wc : 0, c = valid ? gl - pl * P.wc : 0;
  const Axis& ay = P.ay;
  const int r0 = ay.r0, r1 = ay.r1;
  float2* Tl = T + l;
  const float2* wl = P.ws + ((size_t)pl * P.hh) * P.wp + 2 * c;
  float* mats = (float*)(T + ((size_t)P.h << sh));
  if constexpr (MP > 0) copy_matrices<MP>(mats, ay);
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
      if (self) {            // warp-uniform: k0 = 0 or R0 / 2 is its own mirror
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
#pragma unroll
        for (int j2 = 0; j2 < JH; ++j2) {
          const float ax_ = v2x(u[j2]), ay_ = v2y(u[j2]);
          const float wx = __shfl_xor_sync(0xffffffffu, ax_, NL);
          const float wy = __shfl_xor_sync(0xffffffffu, ay_, NL);
          if (R - 1 - j2 != j2) {
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
  IO* op = (IO*)P.out + (size_t)(P.plane0 + pl) * P.OH * P.OW;
  float2* rl = (float2*)P.r + (size_t)pl * P.h * P.wc + c;
  if constexpr (MP == 0) {
    if (!valid) return;
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
    const int st = r1 << sh;
    matrix_stage<MP>(r0, st, st, mats, [&](int v) { return T + v; });
    __syncthreads();
    if (!valid) return;
    // rows q and r0 - q of a column pair from the same two cells
    const int nq = (r0 / 2 + 1) * r1;
    for (int it = tid >> sh; it < nq; it += nthr >> sh) {
      int q, j;
      divmod_small(it, r1, ay.inv_r1, q, j);
      const float2* x = Tl + (j << sh);
      const float2 a = x[q * st];
      const bool self = q == 0 || 2 * q == r0;
      const float2 b = self ? make_float2(0.f, 0.f) : x[(r0 - q) * st];
      const float2 z0 = make_float2(a.x + b.y, a.y - b.x), z1 = make_float2(a.x - b.y, a.y + b.x);
      const int y0 = j + r1 * q, y1 = j + r1 * (r0 - q);
      if (P.s == 1) {
        store_crop<IO>(P, op, y0, c, z0);
        if (!self) store_crop<IO>(P, op, y1, c, z1);
      } else {
        rl[(size_t)y0 * P.wc] = make_float2(z0.x, -z0.y);
        if (!self) rl[(size_t)y1 * P.wc] = make_float2(z1.x, -z1.y);
      }
    }
  }
}

// ------------------------------------------------------------------ upsampling epilogue of one plane
// out[i][j] = x[i/s][j/s] + sum_{a,b} K[a][b] Z[i+a-c][j+b-c], Z = zero_insert(r) on the circular
// s h x s w grid, cropped.  r: row-major reals, pitch `rp`.  A thread owns CW low-resolution columns and rows
// my0 .. my1 - 1 with a sliding window of r.  `op`: the output plane (direct) or a staged band of it that starts at low
// row `base`.
template <int S, int K, int CW, typename IO>
__device__ __forceinline__ void epi_rows(const Params& P, const float* r, int rp, const float* wk, const IO* xp, IO* op,
                                         int sx, int my0, int my1, int base, bool direct) {
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
  const bool vec = direct && ncell == CW && (oW * (int)sizeof(IO)) % 16 == 0 && (NO * (int)sizeof(IO)) % 16 == 0 &&
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
          if (i + 1 < NO) gelu_fast_pair(oa[i], oa[i + 1]);
          else oa[i] = gelu_erf(oa[i]);
        }
      }
      IO* o = op + (size_t)((my - base) * S + da) * oW + mx0 * S;
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

// n contiguous elements from shared memory; both sides have the same alignment modulo 16 bytes
template <typename IO>
__device__ __forceinline__ void copy_band(IO* to, const IO* from, int n, int t, int items) {
  constexpr int V = 16 / (int)sizeof(IO);
  int head = (int)((16 - ((size_t)to & 15)) & 15) / (int)sizeof(IO);
  if (head > n) head = n;
  const int nv = (n - head) / V;
  for (int i = t; i < nv; i += items) ((uint4*)(to + head))[i] = ((const uint4*)(from + head))[i];
  for (int i = t; i < head; i += items) to[i] = from[i];
  for (int i = head + nv * V + t; i < n; i += items) to[i] = from[i];
}

#define CVB_RP_EPI_CASES(X) X(2, 2, 2, 4) X(2, 3, 2, 4) X(2, 5, 2, 4) X(2, 7, 2, 4) X(3, 3, 4, 4) X(3, 5, 4, 4) X(3, 7, 4, 4) X(4, 3, 1, 2) X(4, 5, 1, 2) X(4, 7, 1, 2)

// rows my0 .. my1 - 1 of one plane by `items` threads with index `t`.  With a band buffer (`band` bytes at `buf`, 16-byte
// aligned, all threads of the block in step) runs that cannot leave as whole 16-byte stores -- odd widths, three bf16
// values a cell -- are collected there row by row and copied out contiguously: 4 x 48 planes of 77 x 118 by 3 in bf16
// spent 75 us of 134 on 2-byte stores 24 bytes apart.
template <typename IO>
__device__ __forceinline__ void epilogue(const Params& P, const float* r, int rp, const float* wk, const IO* xp, IO* op,
                                         int t, int items, int my0, int my1, unsigned char* buf, int band) {
  const int key = P.s * 16 + P.k, oW = P.W * P.s;
  switch (key) {
#define X(S_, K_, CWF, CWB)                                                                             \
  case S_ * 16 + K_: {                                                                                  \
    constexpr int CW = sizeof(IO) == 4 ? CWF : CWB;                                                     \
    const int spr = (P.W + CW - 1) / CW;                                                                \
    const bool aligned = P.W % CW == 0 && (oW * (int)sizeof(IO)) % 16 == 0 &&                           \
                         (CW * S_ * (int)sizeof(IO)) % 16 == 0 && ((size_t)op) % 16 == 0;               \
    if (sizeof(IO) == 4 && S_ == 3 && !aligned) {   /* one cell a lane: neighbouring lanes write neighbouring runs */ \
      const int nseg = items / P.W < 1 ? 1 : items / P.W > my1 - my0 ? my1 - my0 : items / P.W;         \
      const int rps = (my1 - my0 + nseg - 1) / nseg;                                                    \
      for (int i = t; i < P.W * nseg; i += items) {                                                     \
        const int seg = i / P.W, b0 = my0 + seg * rps, b1 = b0 + rps < my1 ? b0 + rps : my1;            \
        if (b0 < b1) epi_rows<S_, K_, S_ == 3 ? 1 : CW, IO>(P, r, rp, wk, xp, op, i - seg * P.W, b0, b1, 0, true); \
      }                                                                                                 \
      break;                                                                                            \
    }                                                                                                   \
    int per = aligned ? 0 : (band - 16) / (S_ * oW * (int)sizeof(IO));   /* low rows of a band */       \
    const bool direct = per < 8 && per < my1 - my0;   /* bands of a few rows leave threads idle */      \
    if (direct) per = my1 - my0;                                                                        \
    for (int m0 = my0; m0 < my1; m0 += per) {                                                           \
      const int m1 = m0 + per < my1 ? m0 + per : my1, rows = m1 - m0;                                   \
      int nseg = items / spr;                                                                           \
      if (nseg < 1) nseg = 1;                                                                           \
      if (nseg > rows) nseg = rows;                                                                     \
      const int rps = (rows + nseg - 1) / nseg;                                                         \
      IO* to = op + (size_t)m0 * S_ * oW;                                                               \
      IO* dst = direct ? op : (IO*)(buf + ((size_t)to & 15));                                           \
      for (int i = t; i < spr * nseg; i += items) {                                                     \
        const int seg = i / spr, sx = i - seg * spr;                                                    \
        const int b0 = m0 + seg * rps, b1 = b0 + rps < m1 ? b0 + rps : m1;                              \
        if (b0 < b1) epi_rows<S_, K_, CW, IO>(P, r, rp, wk, xp, dst, sx, b0, b1, direct ? 0 : m0, direct); \
      }                                                                                                 \
      if (!direct) {                                                                                    \
        __syncthreads();                                                                                \
        copy_band<IO>(to, dst, rows * S_ * oW, t, items);                                               \
        __syncthreads();                                                                                \
      }                                                                                                 \
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
  if (P.s > 1)
    for (int i = tid; i < P.k * P.k; i += nthr) wk[i] = P.weight[(size_t)ch * P.k * P.k + i];
  for (int y = tid; y < h; y += nthr) rowoff[y] = row_offset(P, y);
  __syncthreads();
  // ---- columns forward
  {
    const int r0 = ay.r0, r1 = ay.r1, st = r1 * wc;
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
            float2* Tk = T2 + row * pitch + k0 * r1;
            float re[R], im[R];
#pragma unroll
            for (int j = 0; j < R; ++j) {
              const float2 v = Tk[j];
              re[j] = v.x; im[j] = v.y;
            }
            rows_mid<R>(P, re, im, Tk, tab + row, k0);
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
    if (P.s > 1) {
      __syncthreads();
      if (P.rsave) {
        float2* keep = (float2*)P.rsave + (size_t)plane * h * wc;
        for (int i = tid; i < h * wc; i += nthr) keep[i] = T1[i];
      }
      epilogue<IO>(P, (const float*)T1, 2 * wc, wk, xp, op, tid, nthr, 0, P.H, (unsigned char*)(((size_t)T2 + 15) & ~(size_t)15),
                   hh * pitch * (int)sizeof(float2) - 16);
    }
  }
}

// upsampling epilogue of the multi-launch form: grid (row segments, planes); `buf` holds a band of one segment or less
constexpr int kEpiRows = 16;
constexpr int kEpiBand = 40 * 1024;
template <typename IO>
__device__ __forceinline__ void epilogue_body(const Params& P, unsigned char* buf) {
  const int pl = blockIdx.y, plane = P.plane0 + pl, ch = plane % P.C;
  const int my0 = blockIdx.x * kEpiRows, my1 = my0 + kEpiRows < P.H ? my0 + kEpiRows : P.H;
  epilogue<IO>(P, P.r + (size_t)pl * P.h * P.wp, P.wp, P.weight + (size_t)ch * P.k * P.k,
               (const IO*)P.x + (size_t)plane * P.H * P.W, (IO*)P.out + (size_t)plane * P.H * P.W * P.s * P.s,
               threadIdx.x, blockDim.x, my0, my1, buf, kEpiBand);
}

}  // namespace rp
}  // namespace cvb
