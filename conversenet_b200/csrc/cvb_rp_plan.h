// Host side of the real-plane kernels (cvb_rp.cuh): axis plans, table layout, launch geometry.  Allocates nothing.
#pragma once
#include "cvb_plan.h"
#include "cvb_fix.cuh"

namespace cvb {
namespace rp {

constexpr int kMatrixMax = 127;   // largest R0 of the matrix stage
constexpr int kMatrixN = 1300;    //   and the longest axis whose tile and matrices fit shared memory
constexpr int kMaxR1 = 26;        // (separating the spectra keeps 2 R1 values in a thread: small ones are cheaper)

// N = R0 * R1 with the lowest estimated cost per point: packed butterfly operations plus about nine instructions of
// loads, stores and twiddles a stage; a matrix stage costs R0 FMAs a point.  Radices above kSmallRadix take the
// kernels with fewer resident warps.
inline bool axis_plan(int n, int& r0, int& r1) {
  double best = 1e30;
  auto cost = [&](int r) { return 9.0 + kRadixOps[r] * 0.01 + (r > 16 ? 0.25 * (r - 16) : 0.0) + (r > kSmallRadix ? 2.0 : 0.0); };
  for (int b = 1; b <= kMaxR1 && b <= n; ++b) {
    if (n % b || (b > 1 && !register_radix(b))) continue;
    const int a = n / b;
    if (a < 2) continue;
    double c = b == 1 ? 6.0 : cost(b) + (b > 10 ? 0.3 * (b - 10) : 0.0);
    if (register_radix(a)) c += cost(a);
    else if (a <= kMatrixMax && b <= kMatrixR1 && n <= kMatrixN) c += 20.0 + 1.2 * matrix_width(a) * 2;
    else continue;
    if (c < best) { best = c; r0 = a; r1 = b; }
  }
  return best < 1e30;
}

inline bool supported(int h, int w) {
  int a, b;
  return h >= 2 && w >= 2 && axis_plan(h, a, b) && axis_plan(w, a, b);
}

// Axes that carry an operand for the integer contractions
inline bool fix_axis(int n, int r0) { return fix_length(n) && matrix_width(r0) > 0; }

inline int matrix_entries(int r0) { return 2 * (r0 / 2 + 1) * matrix_width(r0); }   // floats, a multiple of 8

// Blob in float2 units: multiplier [C][w][hh]; twiddles of h and of w in natural order (tw), then in position order
// (twy, twx); matrix rows of R0(h) and of R0(w); operands of the integer contractions along h and w
struct Blob { size_t tw, twy, twx, dmy, dmx, fixy, fixx, total; };
inline Blob blob_layout(int C, int h, int w, int r0y, int r0x) {
  Blob b;
  b.tw = (size_t)C * w * (h / 2 + 1);
  b.twy = (b.tw + h + w + 1) & ~(size_t)1;
  b.twx = (b.twy + h + 1) & ~(size_t)1;
  b.dmy = (b.twx + w + 1) & ~(size_t)1;
  b.dmx = b.dmy + matrix_entries(r0y) / 2;
  b.fixy = (b.dmx + matrix_entries(r0x) / 2 + 1) & ~(size_t)1;
  b.fixx = b.fixy + (fix_axis(h, r0y) ? fix_bytes(h) / 8 : 0);
  b.total = b.fixx + (fix_axis(w, r0x) ? fix_bytes(w) / 8 : 0);
  return b;
}

inline void fill_axis(Axis& a, int n, int r0, int r1, const float2* tw, const float2* dm) {
  a.n = n; a.r0 = r0; a.r1 = r1;
  a.mp = matrix_width(r0);
  a.inv_r1 = 1.0f / (float)r1;
  a.tw = tw; a.dm = (const float*)dm; a.fix = nullptr;
}

inline size_t cols_smem(const Params& P) {
  return (size_t)P.h * kLines * sizeof(float2) + (size_t)((P.h + 3) & ~3) * sizeof(int) +
         (P.ay.mp ? matrix_entries(P.ay.r0) : 0) * sizeof(float);
}
inline size_t rows_smem(const Params& P) {
  return (((size_t)P.pitch * kLines + 1) & ~(size_t)1) * sizeof(float2) + (P.ax.mp ? matrix_entries(P.ax.r0) : 0) * sizeof(float);
}
// kernels built for small radices serve an axis whose two radices are small
inline bool small_axis(const Axis& a) { return a.mp == 0 && a.r0 <= kSmallRadix && a.r1 <= kSmallRadix; }

// Block size of the strip kernels.  Without a matrix stage a stage of a tile is a number of register transforms that the
// threads take in turns, so that a size that divides them badly leaves threads idle for most of the last turn (320 transforms:
// three turns of 128 threads, two of 160), and a larger one fits an SM less often.  Every turn waits for its loads, whatever
// the number of warps; so the size is chosen by the turns of a tile, each weighted with its radix (the ten stand for the
// latency), times the rounds of blocks over the SMs (one at least).  The size to start from is 256 threads where the blocks
// leave SMs idle or where four tiles do not fit an SM's memory, else 128 -- the only sizes of a kernel with a matrix stage --
// and another has to win by a tenth.  Against the times of 96 to 256 threads on 60 kernels and shapes (100 to 512 points, 64 to
// 1024 planes) the choice is within 4 % of the best on average, the start 18 %; the worst is 5 % slower than the start.
// 1 x 64 planes of 240 x 160 75 -> 47 us, of 260 x 340 134 -> 85, rows of 1 x 128 planes of 244 x 324 61 -> 49.
inline int strip_threads(const Params& P, bool rows, int grid, int sms) {
  const Axis& a = rows ? P.ax : P.ay;
  const size_t smem = rows ? rows_smem(P) : cols_smem(P);
  const int start = grid <= 2 * sms || 4 * (smem + 1024) > kSmemLimit + 1024 ? 256 : 128;
  if (a.mp) return start;
  const int registers = small_axis(a) ? 80 : 128;        // of the kernels' launch bounds
  auto turns = [](int n, int t) { return (n + t - 1) / t; };
  int best = start;
  double least = 1e30;
  for (int t = 256; t >= 96; t -= 32) {
    const int resident = (int)((kSmemLimit + 1024) / (smem + 1024)), fit = 65536 / (registers * t);
    const double load = (double)grid / ((double)sms * (resident < fit ? resident : fit));
    const double tile = rows ? 2.0 * turns(a.r1 * kLines, t) * (a.r0 + 10) + turns(a.r0 * kLines, t) * (2 * a.r1 + 10)
                             : turns(a.r1 * kLines, t) * (a.r0 + 10) + turns(a.r0 / 2 + 1, t / (2 * kLines)) * (a.r1 + 10);
    const double cost = tile * (load > 1.0 ? load : 1.0) * (t == start ? 1.0 : 1.1);
    if (cost < least) { least = cost; best = t; }
  }
  return best;
}

inline size_t plane_smem(int h, int w, int k) {
  const int wc = (w + 1) / 2, hh = h / 2 + 1;
  return ((size_t)h * wc + (size_t)hh * (w | 1) + (k * k + 1) / 2) * sizeof(float2) + (size_t)h * sizeof(int);
}

// Everything of Params that depends on the shape; false when an axis has no plan.
inline bool fill_params(Params& P, const void* table, int B, int C, int H, int W, int k, int s, int p, int pad_mode) {
  const int h = H + 2 * p, w = W + 2 * p;
  int r0y, r1y, r0x, r1x;
  if (h < 2 || w < 2 || !axis_plan(h, r0y, r1y) || !axis_plan(w, r0x, r1x)) return false;
  const float2* t = (const float2*)table;
  const Blob bl = blob_layout(C, h, w, r0y, r0x);
  P.tab = t;
  P.B = B; P.C = C; P.H = H; P.W = W; P.k = k; P.s = s; P.p = p; P.pad_mode = pad_mode;
  P.h = h; P.w = w; P.hh = h / 2 + 1; P.wc = (w + 1) / 2; P.wp = 2 * P.wc;
  P.pitch = w | 1;
  P.inv_wc = 1.0f / (float)P.wc; P.inv_hh = 1.0f / (float)P.hh;
  fill_axis(P.ay, h, r0y, r1y, t + bl.twy, t + bl.dmy);
  fill_axis(P.ax, w, r0x, r1x, t + bl.twx, t + bl.dmx);
  if (fix_axis(h, r0y)) P.ay.fix = (const unsigned char*)(t + bl.fixy);
  if (fix_axis(w, r0x)) P.ax.fix = (const unsigned char*)(t + bl.fixx);
  P.status = nullptr;
  P.gelu = 0; P.conj = 0; P.plane0 = 0; P.nplane = 0; P.vec = 0; P.vec_out = 0; P.po = p; P.OH = H; P.OW = W; P.rsave = nullptr;
  P.ws = nullptr; P.r = nullptr; P.x = nullptr; P.out = nullptr; P.weight = nullptr;
  return true;
}

// Strip kernels (kFixFwd, kFixRows, kFixInv) that run as integer contractions (cvb_fix.cuh): along axes that would need a
// matrix stage, from the number of lines on that gives 55 of 100 SMs a tile (a launch takes as long with fewer).  Matrix
// stage / contractions on all three kernels, us, planes of N x N: 244 48 planes (91 tiles) 68.3 / 55.1, 32 planes 42.6 / 51 or
// more; 80 planes (153 tiles, two rounds) 114 / 101; 128 planes of 268 156 / 142, 218 157 / 100, 178 120 / 79.5, 134 48.8 / 40.7;
// 64 planes of 134 (67 tiles) 33.8 / 38 or more.  Wide matrix stages (R0 > 88) lose to any number of lines: 8 planes of 202
// 53.5 / 49.7.  The narrowest (R0 = 37, 41) keep the rows below 240: matrix stages / columns alone / all three, 128 planes of 164
// 71.4 / 69.1 / 77.9, 222 110 / 99.0 / 101, 246 126 / 108.5 / 108.3 (512 planes 513 / 434 / 428).  Register radices
// stay: 128 planes of 264 79 / 124.
inline bool takes_fix(const Params& P, int kind, int sms) {
  const Axis& a = kind == kFixRows ? P.ax : P.ay;
  if (!a.fix || (kind == kFixRows && a.mp <= 20 && a.n < 240)) return false;
  const long long tiles = (fix_lines(kind, P) + kFixLines - 1) / kFixLines;
  return a.mp >= 56 || 100 * tiles >= 55 * (long long)sms;
}

// Bytes of workspace one plane takes in the multi-launch form
inline size_t ws_plane_bytes(int h, int w, int s) {
  const int wp = (w + 1) / 2 * 2;
  const size_t spec = (size_t)(h / 2 + 1) * wp * sizeof(float2);
  return s > 1 ? spec + ((size_t)h * wp * sizeof(float) + 15) / 16 * 16 : spec;
}

// One block per plane (plane_body) or three launches, by the shared memory a plane takes:
//   more planes than SMs: while three planes share an SM's memory
//   no more planes than SMs, a block of up to 512 threads each: up to 96 KB; up to 148 KB when the planes occupy two
//   thirds of the SMs, because the time of the launches grows with the planes and that of the block does not
// (one block / three launches, us at scale 1, planes per call: 28 x 24, 16 6.4 / 8.8; 76 x 76, 47 KB, 64 13.3 / 18.1,
// 148 13.5 / 21.6; 108 x 108, 94 KB, 16 13.7 / 14.7, 148 14.1 / 23.9; 132 x 132, 139 KB, 64 20.5 / 17.9, 128 20.6 / 26.9)
constexpr size_t kPlaneThree = 75 * 1024, kPlaneWide = 96 * 1024, kPlaneMost = 148 * 1024;
inline size_t one_block_limit(int planes, int sms) {
  return planes > sms ? kPlaneThree : 3 * planes >= 2 * sms ? kPlaneMost : kPlaneWide;
}

struct Route {
  bool one_block;       // plane_body, no workspace
  int threads;          //   its block size
  int chunk;            // multi-launch form: planes per chunk
  size_t ws_bytes;
};
// One block per plane up to one_block_limit, else the multi-launch form over chunks of at most ws_cap bytes of workspace.
inline Route route(int B, int C, int H, int W, int s, int p, int sms, bool force_multi, size_t ws_cap) {
  const int h = H + 2 * p, w = W + 2 * p, planes = B * C;
  Route r;
  const size_t sm = plane_smem(h, w, kMaxTaps);
  int a, b, c, d;
  axis_plan(h, a, b);
  axis_plan(w, c, d);
  r.one_block = !force_multi && register_radix(a) && register_radix(c) && sm <= one_block_limit(planes, sms);
  r.threads = 256;
  const size_t per = ws_plane_bytes(h, w, s);
  size_t n = ws_cap / per;
  if (n > (size_t)planes) n = planes;
  if (n > 0) {                            // chunks of equal size, as many as
    const int least = (planes + (int)n - 1) / (int)n;
    const bool fy = fix_axis(h, a), fx = fix_axis(w, c);
    // rounds of tiles that the integer contractions take for m planes: 4 x 128 planes of 268 x 268 in four chunks (two rounds
    // a kernel each) take 0.91 of the time in three (2.4, that is three)
    auto rounds = [&](int m) {
      auto of = [&](long long lines) { return (int)((lines + (long long)kFixLines * sms - 1) / ((long long)kFixLines * sms)); };
      return (fy ? 2 * of((long long)m * (w + 1)) : 0) + (fx ? 2 * of(2LL * m * (h / 2 + 1)) : 0);
    };
    int best = least, most = 0x7fffffff;
    for (int q = least; q < least + 4 && (q == least || ((fy || fx) && q <= planes)); ++q) {
      const int m = (planes + q - 1) / q, whole = planes / m, total = whole * rounds(m) + (planes % m ? rounds(planes % m) : 0);
      if (total < most) { most = total; best = q; }
    }
    n = (planes + best - 1) / best;
  }
  r.chunk = (int)n;
  r.ws_bytes = r.one_block ? 0 : n * per;
  return r;
}

// Block size of plane_body.  Planes enough to fill the SMs: the count that wastes the fewest thread slots over the
// stages.  Fewer: the count with the shortest chain of stage passes.
inline int plane_threads(const Params& P, int most, bool fills) {
  const Axis &y = P.ay, &x = P.ax;
  const int items[4] = {y.r1 * P.wc, (y.r0 / 2 + 1) * P.wc, x.r1 * P.hh, x.r0 * P.hh};
  const int cost[4] = {y.r0, 2 * y.r1, x.r0, x.r1};
  double best = 1e30;
  int bt = 64;
  for (int t = 64; t <= most; t += 32) {
    double c = 0;
    for (int i = 0; i < 4; ++i) c += (double)((items[i] + t - 1) / t) * (cost[i] + (fills ? 2 : 8));
    c *= fills ? t * (1.0 + 8.0 / t) : 1.0 + t / 4096.0;      // (fewer warps hide less latency; more wait longer)
    if (c < best - 1e-9) { best = c; bt = t; }
  }
  return bt;
}

}  // namespace rp
}  // namespace cvb
