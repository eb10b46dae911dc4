// The strip kernels of the real-plane solve (cvb_rp.cuh) as integer contractions on the tensor cores: any even length
// N = 2 M from 130 to 270, whatever its prime factors.
//
// A real line x_0 .. x_(N-1) folds into four sums per q = 0 .. M / 2,
//     a = x_q + x_(M+q),  b = x_(N-q) + x_(M-q),  c = x_q - x_(M+q),  d = x_(N-q) - x_(M-q),
// and its transform X_k = C_k - i S_k is a product with a constant matrix per parity of k:
//     C_k = sum_q cos(2 pi k q / N) u_q,   S_k = sum_q sin(2 pi k q / N) v_q,   k <= M,
//     k even: u = a + b, v = a - b;   k odd: u = c + d, v = c - d    (weight 1/2 at q = 0 and q = M / 2, counted twice).
// A complex row is two real lines; the inverse along the columns starts from lines that are folded already.
//
// Arithmetic.  A line is scaled by a power of two so that its sums u and v stay below 2^30 and these are rounded to 32-bit
// integers, cut into four signed base-256 digits; the constants are 24-bit integers, three digits.  Products of digits
// accumulate exactly in 32-bit integers (tcgen05.mma kind::i8), one accumulator per weight 256^-(i + j), i + j <= 3; what
// is left out lies 2^-32 below the largest value.  So the only roundings are those of the constants (2^-24), the folds and
// the result: 1.8e-7 of a 268 x 268 plane's norm against fp64, where fp32 butterflies and dense stages are at 2.2e-7 or
// more, whatever the magnitude of a line (one whose largest value is below 2^-87 takes its scale in two steps).  A line
// with an infinity or a NaN becomes NaN, and with it, as in any transform, its plane.
//
// One block per SM walks over tiles of 128 lines (= rows of the MMA = lanes of tensor memory).  A tile arrives in shared
// memory as it is; thread t serves line t % 128: it folds a quarter of the line's q, cuts the four classes into digits and
// writes them to tensor memory (256 columns), from where the MMAs read them.  The constants' digits lie side by side along N
// in shared memory (36 to 60 KB), and so do the accumulators; a pair of digits is an MMA.  Outputs come in chunks of 32
// frequencies of one parity, cosines and sines (what 32 does not divide: 16 of both parities), in the other 256 columns of tensor
// memory; a thread reads back eight frequencies of its line.  The warp that is the last to have read a chunk issues the MMAs of
// the next one, which run while the values are finished and stored.
// q >= 64 (lengths from 256 on: at most four) is added in fp32 there.
// Columns: the next tile is copied to shared memory as soon as the last one is folded.  Rows: the forward transform, the
// multiplier and the transform back follow each other on a tile that stays in shared memory.
//
// What bounds it: a chain per chunk (MMAs issued one after the other, their latency, tensor memory read, converted) at four warps a
// scheduler; half of the issue slots and a tenth of the tensor pipe are used.  1 x 128 planes of 268 x 268: 140 us, with the
// matrix stages 156; 244 x 244 105 / 138; 178 x 178 77 / 120; 254 x 254 (R0 = 127) 106 / 287.
// A digit of the line times several of the constants' as one MMA 3 n, 2 n and n columns wide, four a K step instead of nine, took
// 126, 99, 74 and 100 us, but those overlap in accumulators without the same shape, and nothing orders such MMAs.  Tried with it:
// pairs of accumulators 2 n wide with zeros beside the constants' digits, six a K step 144 us (columns cost more than MMAs);
// cosines and sines by turns 138 against 140, 1 % slower at other lengths.
// Tried on the way (against the 126 us): digits in shared memory 180 us; MMAs issued by a divergent lane instead of a whole warp with
// one lane elected 152; 1024 threads of 64 registers 139; cosines and sines as chunks of their own 203 (with spills); the MMA
// loops unrolled 135 (instruction fetch).
#pragma once
#include "cvb_rp.cuh"
#ifdef __CUDACC__
#include "cvb_tc.cuh"
#else
#include "cvb_tma.cuh"
#endif

namespace cvb {
namespace rp {

enum { kFixFwd = 0, kFixRows = 1, kFixInv = 2 };
constexpr int kFixLines = 128, kFixParts = 4;    // lines of a tile; threads that share the work on a line
constexpr int kFixThreads = kFixParts * kFixLines, kFixWarps = kFixThreads / 32, kFixWait = 1 << 20;
// Constants are stored as rint(value / kFixUnit); the unit is an fp32 number, so that undoing the scale rounds once.
constexpr float kFixUnit = 1.1967864e-07f;       // just above 1 / 0x7f7f7f, the largest number of three signed digits

// ------------------------------------------------------------------ tensor memory, barriers, copies
#ifdef __CUDACC__
__device__ __forceinline__ void fx_alloc(uint32_t* holder) { tc::tmem_alloc(holder, 512); }
__device__ __forceinline__ void fx_free(uint32_t t) { tc::tmem_dealloc(t, 512); }
__device__ __forceinline__ void fx_before_sync() { tc::fence_before_sync(); }
__device__ __forceinline__ void fx_after_sync() { tc::fence_after_sync(); }
__device__ __forceinline__ uint32_t fx_elect() { return tc::elect_one(); }
__device__ __forceinline__ void fx_commit(uint64_t* bar) { tc::mma_commit(bar); }
__device__ __forceinline__ void fx_init(uint64_t* bar) { mbar_init(bar, 1); }
__device__ __forceinline__ void fx_init_done() { mbar_fence_init(); }
__device__ __forceinline__ void fx_expect(uint64_t* bar, uint32_t bytes) { mbar_expect_tx(bar, bytes); }
__device__ __forceinline__ void fx_bulk(void* dst, const void* src, uint32_t bytes, uint64_t* bar) { bulk_g2s(dst, src, bytes, bar); }
__device__ __forceinline__ bool fx_wait(uint64_t* bar, uint32_t parity) { return mbar_wait_bounded(bar, parity, kFixWait); }
// counts an arrival: what happened before it is visible to whom a later arrival finds it counted
__device__ __forceinline__ unsigned fx_count(unsigned* counter) {
  unsigned old;
  asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;" : "=r"(old) : "r"(smem_u32(counter)) : "memory");
  return old;
}
__device__ __forceinline__ unsigned fx_from_first(unsigned v) { return tc::from_first(v); }
// the second operand of fx_mma: rows of 16 bytes, eight of them a core matrix, the second half of K `brows` rows further on
__device__ __forceinline__ uint64_t fx_operand(const unsigned char* b, int brows) { return tc::smem_desc(b, 16 * brows, 128); }
__device__ __forceinline__ uint64_t fx_further(uint64_t b, int bytes) { return b + (uint32_t)(bytes >> 4); }
// D[128 x n] (+)= A[128 x 32] B[n x 32]^T, signed bytes, 32-bit sums.  A: eight columns of tensor memory, four bytes each
__device__ __forceinline__ void fx_mma(uint32_t d, uint32_t a, uint64_t b, int n, bool add, uint32_t elected) {
  const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | (8u << 24);
  asm volatile(
      "{\n\t"
      ".reg .pred p, e;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 e, %5, 0;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t"
      "}\n" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(add ? 1u : 0u), "r"(elected)
      : "memory");
}
// consecutive columns of this thread's lane
__device__ __forceinline__ void fx_ld(uint32_t t, int (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(t) : "memory");
}
__device__ __forceinline__ void fx_ld(uint32_t t, int (&v)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(t) : "memory");
}
__device__ __forceinline__ void fx_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void fx_st(uint32_t t, const uint32_t (&v)[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(t), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
__device__ __forceinline__ void fx_st(uint32_t t, const uint32_t (&v)[2]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(t), "r"(v[0]), "r"(v[1]) : "memory");
}
__device__ __forceinline__ void fx_st_wait() { tc::tmem_wait_st(); }
// asynchronous copies to shared memory; zeros where `ok` is false
template <int BYTES>
__device__ __forceinline__ void fx_copy(void* dst, const void* src, bool ok) {
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(ok ? 16 : 0) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(smem_u32(dst)), "l"(src), "n"(BYTES), "r"(ok ? BYTES : 0) : "memory");
}
__device__ __forceinline__ void fx_copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// the largest magnitude; a NaN stays
__device__ __forceinline__ float fx_largest(float m, float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(m), "f"(fabsf(a)), "f"(fabsf(b)));
  return r;
}
__device__ __forceinline__ float2 fx_fma2(float2 a, float2 b, float2 c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d)
      : "l"(*(const uint64_t*)&a), "l"(*(const uint64_t*)&b), "l"(*(const uint64_t*)&c));
  return *(float2*)&d;
}
__device__ __forceinline__ float2 fx_mul2(float2 a, float2 b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(*(const uint64_t*)&a), "l"(*(const uint64_t*)&b));
  return *(float2*)&d;
}
#endif

// ------------------------------------------------------------------ geometry
// Up to 270: tensor memory holds the digits of that many points.  From 130: where the measurements begin that takes_fix
// (cvb_rp_plan.h) rests on.  The kernel itself is right from 66 on and faster than the matrix stages from about 94 points along
// columns and 118 along rows (128 planes of 122 x 122 34 / 46 us, of 94 x 94 32 / 35; 256 of 300 x 94 124 / 117).
__host__ __device__ constexpr bool fix_length(int n) { return n % 2 == 0 && n >= 130 && n <= 270; }
__host__ __device__ constexpr int fix_rows(int n) { return (n / 4 + 16) & ~15; }       // frequencies of a parity, padded
__host__ __device__ constexpr int fix_operand(int n) { return 768 * fix_rows(n); }     // bytes: 2 parities x 2 x 3 digits x 64
__host__ __device__ constexpr int fix_bytes(int n) { return fix_operand(n) + 64 * fix_rows(n); }   // and fp32 q = 64 .. 67
// where digit 0 of row j, quantity cs (0 cosine, 1 sine) of parity par lies, and how far the next digit is
__host__ __device__ inline int fix_row_offset(int nr, int par, int cs, int j, int q, int& digit_step) {
  const int j0 = j & ~31, n = nr - j0 < 32 ? nr - j0 : 32;
  digit_step = 16 * n;
  return 384 * (par * nr + j0) + cs * 192 * n + (q >> 4) * 48 * n + (j - j0) * 16 + (q & 15);
}
// Shared memory: the tile (128 values for every q, rows: 64 complex ones and one of padding), the constants, extra
// q, largest values (of two passes), barriers, columns forward: where each padded row starts
constexpr int kFixPitch = 65;
__host__ __device__ inline size_t fix_area(int kind, int n) {
  return kind == kFixRows ? ((size_t)8 * kFixPitch * n + 15) / 16 * 16 : kind == kFixInv ? (size_t)1024 * (n / 2 + 1) : (size_t)512 * n;
}
__host__ __device__ inline size_t fix_smem(int kind, int n) {
  return fix_area(kind, n) + fix_bytes(n) + (n >= 256 ? 16 * kFixLines * 4 : 0) + 2 * kFixLines * 4 + 48 +
         (kind == kFixFwd ? (size_t)(n + 4) * 4 : 0);
}
// Lines of a launch: columns forward, all columns of the workspace; rows, two lines each; columns inverse, the columns
// that are kept
__host__ __device__ inline int fix_columns(int kind, const Params& P) { return kind == kFixInv && P.s == 1 ? P.OW : P.wp; }
__host__ __device__ inline int fix_lines(int kind, const Params& P) {
  return P.nplane * (kind == kFixRows ? 2 * P.hh : fix_columns(kind, P));
}

// what a line's scale 2^(29 - exponent), 2^116 at most, lacks for its largest value (its bits) to reach 2^29
__device__ __forceinline__ float fix_rest(unsigned largest) {
  const int ex = (int)(largest >> 23);
  return __uint_as_float((uint32_t)(127 + (ex < 1 ? 39 : ex < 40 ? 40 - ex : 0)) << 23);
}
// a thread's values of a class to tensor memory: Q / 4 columns of each digit
template <int Q>
__device__ __forceinline__ void fix_digits(const float (&v)[Q], float scale, uint32_t t) {
  uint32_t w[4][Q / 4];      // [digit][four q]
#pragma unroll
  for (int g = 0; g < Q / 4; ++g) {
    uint32_t n[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) n[i] = (uint32_t)__float2int_rn(v[4 * g + i] * scale) + 0x80808080u;
    const uint32_t l0 = __byte_perm(n[0], n[1], 0x5140), h0 = __byte_perm(n[0], n[1], 0x7362);
    const uint32_t l1 = __byte_perm(n[2], n[3], 0x5140), h1 = __byte_perm(n[2], n[3], 0x7362);
    w[3][g] = __byte_perm(l0, l1, 0x5410) ^ 0x80808080u;
    w[2][g] = __byte_perm(l0, l1, 0x7632) ^ 0x80808080u;
    w[1][g] = __byte_perm(h0, h1, 0x5410) ^ 0x80808080u;
    w[0][g] = __byte_perm(h0, h1, 0x7632) ^ 0x80808080u;
  }
#pragma unroll
  for (int d = 0; d < 4; ++d) fx_st(t + 16 * d, w[d]);
}

// the MMAs of n frequencies of one class: digits at column a (16 columns each), accumulators at column t.  One for each pair of
// digits (i, j), i + j <= 3, into the accumulator i + j: MMAs keep the order of their issue only among those of the same
// accumulator and shape, so every MMA that meets an accumulator has its columns and no others.
__device__ __forceinline__ void fix_issue(const int n, uint32_t t, uint32_t a, const unsigned char* from, uint32_t elected) {
  const auto b0 = fx_operand(from, 3 * n);
#pragma unroll
  for (int kc = 0; kc < 2; ++kc, a += 8) {
#pragma unroll
    for (int p = 0; p < 9; ++p) {
      // (the four that begin an accumulator first, neighbours on different ones)
      const int i = p < 3 ? 0 : p == 3 ? 3 : p < 7 ? 1 : 2, j = p < 3 ? p : p == 3 ? 0 : p < 7 ? p - 4 : p - 7;
      fx_mma(t + (i + j) * n, a + 16 * i, fx_further(b0, 96 * n * kc + 16 * n * j), n, kc > 0 || p > 3, elected);
    }
  }
}
// chunk `it` of a pass: chunks of 32 (`full` per parity), then the rest of both parities; a whole warp
__device__ __forceinline__ void fix_chunk(uint32_t tm, const unsigned char* B, int NR, int it, uint64_t* done, bool ok) {
  const uint32_t elected = fx_elect();
  fx_after_sync();
  if (ok) {
    const int full = NR >> 5, tail = it >= 2 * full, n = tail ? 16 : 32, par = it >= full, c = it - par * full;
    const unsigned char* b = B + (tail ? 384 * 32 * full : 384 * (par * NR + 32 * c));
#pragma unroll 1
    for (int u = 0; u < (tail ? 4 : 2); ++u)
      fix_issue(n, tm + 256 + 4 * n * u, tm + 64 * u + (tail ? 0 : par * 128), b + (u >> 1) * 384 * NR + (u & 1) * 192 * n, elected);
  }
  if (elected) fx_commit(done);
  __syncwarp();
}

// sums from their accumulators, times `undo`
template <int J>
__device__ __forceinline__ void fix_values(const int (&a)[4][J], float undo, float2 (&v)[J / 2]) {
#pragma unroll
  for (int i = 0; i < J / 2; ++i) {
    const float2 hi = make_float2((float)(a[0][2 * i] * 256 + a[1][2 * i]), (float)(a[0][2 * i + 1] * 256 + a[1][2 * i + 1]));
    const float2 lo = make_float2((float)(a[2][2 * i] * 256 + a[3][2 * i]), (float)(a[2][2 * i + 1] * 256 + a[3][2 * i + 1]));
    v[i] = fx_mul2(fx_fma2(hi, make_float2(65536.f, 65536.f), lo), make_float2(undo, undo));
  }
}

// What a kernel knows of its axis and its shared memory; cheap to make again, so that it need not stay in registers
template <int KIND, bool EXTRA>
struct FixBlock {
  int N, M, QH, NR, full, chunks, per, x0;
  unsigned char* B;
  const float* coef;       // [parity][cosine, sine][extra q][row]
  float* xe;               // [class][extra q][line]
  unsigned* largest;       // [2][line]
  uint64_t* done;          // a chunk's MMAs; the constants' arrival
  unsigned* counter;       // warps that have read a chunk
  uint32_t* holder;
  int* rowoff;
  __device__ __forceinline__ FixBlock(const Params& P, unsigned char* smem) {
    N = KIND == kFixRows ? P.ax.n : P.ay.n;
    M = N >> 1; QH = M >> 1; NR = fix_rows(N); full = NR >> 5; chunks = 2 * full + ((NR >> 4) & 1);
    per = KIND == kFixRows ? 2 * P.hh : fix_columns(KIND, P);
    x0 = KIND == kFixInv && P.s == 1 ? P.po : 0;
    B = smem + fix_area(KIND, N);
    coef = (const float*)(B + fix_operand(N));
    xe = (float*)(B + fix_bytes(N));
    largest = (unsigned*)(xe + (EXTRA ? 16 * kFixLines : 0));
    done = (uint64_t*)(largest + 2 * kFixLines);
    counter = (unsigned*)(done + 3);
    holder = (uint32_t*)(counter + 3);
    rowoff = (int*)(done + 6);
  }
};

// Columns: slice `sl` of `ns` of a tile on its way to shared memory: fp32 and the spectra by asynchronous copies, bf16 by plain
// loads and stores (the copies do not convert)
template <int KIND, typename IO, bool EXTRA>
__device__ __forceinline__ void fix_load(const Params& P, unsigned char* smem, int tile, int sl, int ns) {
  const FixBlock<KIND, EXTRA> S(P, smem);
  const int tid = threadIdx.x, per = S.per, lines = fix_lines(KIND, P), first = tile * kFixLines / per;
  const bool pairs = KIND == kFixInv ? ((S.x0 | per) & 1) == 0 : sizeof(IO) == 4 && P.vec && P.pad_mode != 3;   // two columns at once
  const int l = pairs ? 2 * (tid & 63) : tid & (kFixLines - 1), step = pairs ? kFixThreads / 64 : kFixParts, mine = pairs ? tid >> 6 : tid >> 7;
  const int gl = tile * kFixLines + l, pl = gl < lines ? gl / per : first, x = gl - pl * per + S.x0;
  if (KIND == kFixInv) {
    if (gl >= lines) return;
    const float2* src = P.ws + (size_t)first * P.hh * P.wp + (uint32_t)((pl - first) * P.hh * P.wp + x);
    unsigned char* dst = smem + l * 8;
    const int k1 = (S.M + 1) * (sl + 1) / ns;
    int k = (S.M + 1) * sl / ns + mine;
    if (pairs)
      for (; k < k1; k += step) fx_copy<16>(dst + k * (kFixLines * 8), src + (uint32_t)(k * P.wp), true);
    else
      for (; k < k1; k += step) fx_copy<8>(dst + k * (kFixLines * 8), src + (uint32_t)(k * P.wp), true);
  } else {
    const int c = gl < lines && x < P.w ? pad_index(x - P.p, P.W, P.pad_mode) : -1;
    const char* src = (const char*)((const IO*)P.x + (size_t)(P.plane0 + first) * P.H * P.W);
    const int off = c < 0 ? 0 : ((pl - first) * P.H * P.W + c) * (int)sizeof(IO);
    unsigned char* dst = smem + l * 4;
    const int y1 = S.N * (sl + 1) / ns;
    int y = S.N * sl / ns + mine;
    const int c1 = pairs ? pad_index(x + 1 - P.p, P.W, P.pad_mode) : 0;
    if (pairs && (c < 0 || c + 1 == c1)) {      // (neighbours in x as well, or none)
      for (; y < y1; y += step) fx_copy<8>(dst + y * (kFixLines * 4), src + (uint32_t)(off + S.rowoff[y]), c >= 0);
    } else {
      for (; y < y1; y += step) {
        const int o = S.rowoff[y];
        const bool in = c >= 0 && o >= 0;
        if constexpr (sizeof(IO) == 4) {
          fx_copy<4>(dst + y * (kFixLines * 4), src + (uint32_t)(in ? off + o : 0), in);
          if (pairs) fx_copy<4>(dst + y * (kFixLines * 4) + 4, src + (uint32_t)(off + (c1 - c) * 4 + o), true);
        } else {
          *(float*)(dst + y * (kFixLines * 4)) = in ? ld_io<IO>(src + (uint32_t)(off + o), 0) : 0.f;
        }
      }
    }
  }
}
// Rows: a finished tile (if any) goes out, the next one (if any) comes in, row by row, each value by the same thread
__device__ __forceinline__ void fix_exchange(const Params& P, unsigned char* smem, int out, int in, int tiles) {
  const int lane = threadIdx.x & 31, last = P.nplane * P.hh, N = P.ax.n;
  for (int r = threadIdx.x >> 5; r < 64; r += kFixWarps) {
    float2* at = (float2*)smem + r;
    if (out >= 0 && out * 64 + r < last) {
      float2* dst = P.ws + (size_t)(out * 64 + r) * P.wp;
      for (int x = lane; x < N; x += 32) dst[x] = at[x * kFixPitch];
    }
    if (in < tiles && in * 64 + r < last) {
      const float2* src = P.ws + (size_t)(in * 64 + r) * P.wp;
      for (int x = lane; x < N; x += 32) fx_copy<8>(at + x * kFixPitch, src + x, true);
    }
  }
}

template <int KIND, typename IO, bool EXTRA>
__device__ __forceinline__ void fix_body(const Params& P, unsigned char* smem) {
  constexpr int QP = 64 / kFixParts, JP = 32 / kFixParts, TP = kFixParts / 4;     // q, frequencies of a chunk; tail groups
  const int tid = threadIdx.x, lane = tid & 31, warp = (int)fx_from_first(tid >> 5);
  const FixBlock<KIND, EXTRA> S(P, smem);
  const int N = S.N, M = S.M, QH = S.QH, full = S.full, chunks = S.chunks, per = S.per;
  const int lines = fix_lines(KIND, P), tiles = (lines + kFixLines - 1) / kFixLines;

  if (tid == 0) {
    fx_init(S.done); fx_init(S.done + 1);
    fx_init_done();
    fx_expect(S.done + 1, fix_bytes(N));
    fx_bulk(S.B, KIND == kFixRows ? P.ax.fix : P.ay.fix, fix_bytes(N), S.done + 1);
    S.counter[0] = 0;
  }
  if (warp == 0) fx_alloc(S.holder);
  if (tid < 2 * kFixLines) S.largest[tid] = 0;
  if (KIND == kFixFwd)       // in bytes; -1: zeros
    for (int y = tid; y < N; y += kFixThreads) {
      const int o = row_offset(P, y);
      S.rowoff[y] = o < 0 ? -1 : o * (int)sizeof(IO);
    }
  fx_before_sync();
  __syncthreads();
  fx_after_sync();
  const uint32_t tm = fx_from_first(*S.holder);

  const int line = tid & (kFixLines - 1), part = warp >> 2, q0 = part * QP;    // part: which share of the work on the line
  const uint32_t lane_base = tm + ((uint32_t)(warp & 3) << 21);
  constexpr float kTwice = KIND == kFixRows ? 1.f : 2.f;
  const bool mirror = KIND == kFixRows && (line & 1);

  if (KIND == kFixRows) fix_exchange(P, smem, -1, blockIdx.x, tiles);
  else if ((int)blockIdx.x < tiles) fix_load<KIND, IO, EXTRA>(P, smem, blockIdx.x, 0, 1);
  bool ok = fx_wait(S.done + 1, 0);
  uint32_t number = 0, flip = 0;       // chunks so far; which array of largest values

  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int gl = tile * kFixLines + line;
    const bool valid = gl < lines;
    // columns: plane and column of the line; rows: row 64 tile + line / 2, part line & 1.  Addresses are 32-bit offsets
    // from the tile's first plane.
    const int first = tile * kFixLines / per;
    const int pl = valid ? gl / per : first;
    const int at = valid ? KIND == kFixRows ? (gl - pl * per) >> 1 : gl - pl * per + S.x0 : S.x0;

    for (int pass = 0; pass < (KIND == kFixRows ? 2 : 1); ++pass) {
      unsigned* largest = S.largest + flip * kFixLines + line;
      const float* rl = (const float*)smem + (KIND == kFixInv ? line * 2 : line);
      if (pass == 0) fx_copies_done();
      __syncthreads();                   // the tile has arrived; the pass before is over
      // ---- the line's classes, their largest magnitude ----
      // nq: N - q, or 0 for q = 0
      auto fold = [&](int q, int nq, float& v0, float& v1, float& v2, float& v3) {
        if (KIND == kFixInv) {
          const float2 u = *(const float2*)(rl + q * 256), w = *(const float2*)(rl + (M - q) * 256);
          v0 = u.x + w.x; v1 = u.y - w.y; v2 = u.x - w.x; v3 = u.y + w.y;
        } else {
          constexpr int st = KIND == kFixRows ? 2 * kFixPitch : kFixLines;
          const float x0 = rl[st * q], x1 = rl[st * (M + q)], x2 = rl[st * nq], x3 = rl[st * (M - q)];
          const float a = x0 + x1, b = x2 + x3, c = x0 - x1, d = x2 - x3;
          v0 = a + b; v1 = a - b; v2 = c + d; v3 = c - d;
        }
      };
      float v[4][QP];
      if (q0 <= QH) {
        fold(q0, q0 ? N - q0 : 0, v[0][0], v[1][0], v[2][0], v[3][0]);
#pragma unroll
        for (int i = 1; i < QP; ++i) fold(q0 + i, N - q0 - i, v[0][i], v[1][i], v[2][i], v[3][i]);
        float m = 0.f;
#pragma unroll
        for (int i = 0; i < QP; ++i) m = fx_largest(fx_largest(m, v[0][i], v[1][i]), v[2][i], v[3][i]);
        atomicMax(largest, __float_as_uint(m));
      }
      if (EXTRA) {
        float e[4] = {0.f, 0.f, 0.f, 0.f};
        if (64 + part <= QH) fold(64 + part, N - 64 - part, e[0], e[1], e[2], e[3]);
#pragma unroll
        for (int c = 0; c < 4; ++c) S.xe[(c * 4 + part) * kFixLines + line] = kTwice * e[c];
      }
      __syncthreads();                   // the tile has been read
      if (KIND != kFixRows && tile + (int)gridDim.x < tiles) fix_load<KIND, IO, EXTRA>(P, smem, tile + gridDim.x, 0, 1);
      // ---- digits ----
      int ex = (int)(*largest >> 23);
      const bool bad = ex >= 255;
      const bool tiny = __any_sync(0xffffffffu, ex < 40 && *largest != 0);            // somewhere in the warp
      ex = ex < 40 ? 40 : ex > 254 ? 254 : ex;
      const float scale = __uint_as_float((uint32_t)(283 - ex) << 23);             // 2^(29 - exponent)
      if (tiny) {
        const float rest = fix_rest(*largest);
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < QP; ++i) v[c][i] *= rest;
      }
      // x = n / scale, constant = m * unit, the accumulators' lowest weight is 2^16
      const float undo = bad ? __uint_as_float(0x7fc00000u) : kTwice * (kFixUnit * 65536.f) * __uint_as_float((uint32_t)(ex - 29) << 23);
      if (q0 <= QH) {
#pragma unroll
        for (int c = 0; c < 4; ++c) fix_digits<QP>(v[c], scale, lane_base + (uint32_t)(c * 64 + part * (QP / 4)));
        fx_st_wait();
      }
      flip ^= 1;
      if (part == 0) S.largest[flip * kFixLines + line] = 0;        // of the pass before; the next one's
      fx_before_sync();
      __syncthreads();                   // the digits are there
      if (warp == (int)(number & (kFixWarps - 1))) fix_chunk(tm, S.B, S.NR, 0, S.done, ok);      // the warps take turns

      // ---- read-back ----
      for (int it = 0; it < chunks; ++it, ++number) {
        const bool tail = it >= 2 * full;
        const int sub = tail ? part & (2 * TP - 1) : part;                // this thread's group of JP frequencies
        const int par = tail ? part / (2 * TP) : it >= full, n = tail ? 16 : 32;
        const int j0 = 32 * (tail ? full : it - par * full) + JP * sub, k0 = 2 * j0 + par;
        const bool any = k0 <= M;
        float2 gt[JP];
        if (KIND == kFixRows && pass == 0 && any) {       // (asked for before the wait)
          const float2* tab = P.tab + (size_t)((P.plane0 + pl) % P.C) * P.w * P.hh + at;
#pragma unroll
          for (int i = 0; i < JP; ++i) {
            const int k = k0 + 2 * i < M ? k0 + 2 * i : M;
            gt[i] = __ldg(tab + (uint32_t)((mirror && k ? N - k : k) * P.hh));
          }
        }
        float2 C[JP / 2], D[JP / 2];
        if (ok) ok = fx_wait(S.done, number & 1);
        fx_after_sync();
        if (any) {
          const uint32_t t = lane_base + (uint32_t)(256 + (tail ? par * 128 : 0) + JP * sub);
          int acc[4][JP];
#pragma unroll
          for (int i = 0; i < 4; ++i) fx_ld(t + i * n, acc[i]);
          fx_ld_wait();
          fix_values<JP>(acc, undo, C);
#pragma unroll
          for (int i = 0; i < 4; ++i) fx_ld(t + (4 + i) * n, acc[i]);
          fx_ld_wait();
          fx_before_sync();
          fix_values<JP>(acc, undo, D);
          if (tiny) {
            const float back = 1.f / fix_rest(S.largest[(flip ^ 1) * kFixLines + line]);
#pragma unroll
            for (int i = 0; i < JP / 2; ++i) {
              C[i] = fx_mul2(C[i], make_float2(back, back));
              D[i] = fx_mul2(D[i], make_float2(back, back));
            }
          }
        }
        __syncwarp();
        if (it + 1 < chunks) {
          unsigned arrived = 0;
          if (lane == 0) arrived = fx_count(S.counter);
          arrived = fx_from_first(arrived);
          // the last warp to have read the chunk issues the next one
          if ((arrived & (kFixWarps - 1)) == kFixWarps - 1) fix_chunk(tm, S.B, S.NR, it + 1, S.done, ok);
        }
        if (!any) continue;

        if (EXTRA) {
          const float* x = S.xe + par * 8 * kFixLines + line;
          const float* f = S.coef + par * 8 * S.NR + j0;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float a = x[u * kFixLines], b = x[(4 + u) * kFixLines];
#pragma unroll
            for (int i = 0; i < JP / 4; ++i) {
              const float4 fc = *(const float4*)(f + u * S.NR + 4 * i), fs = *(const float4*)(f + (4 + u) * S.NR + 4 * i);
              C[2 * i] = fx_fma2(make_float2(fc.x, fc.y), make_float2(a, a), C[2 * i]);
              C[2 * i + 1] = fx_fma2(make_float2(fc.z, fc.w), make_float2(a, a), C[2 * i + 1]);
              D[2 * i] = fx_fma2(make_float2(fs.x, fs.y), make_float2(b, b), D[2 * i]);
              D[2 * i + 1] = fx_fma2(make_float2(fs.z, fs.w), make_float2(b, b), D[2 * i + 1]);
            }
          }
        }
        if (KIND == kFixFwd) {
          char* base = (char*)(P.ws + (size_t)first * P.hh * P.wp);
          const uint32_t row = (uint32_t)P.wp * 16, to = (uint32_t)((pl - first) * P.hh * P.wp + at + k0 * P.wp) * 8;
          if (valid) {
#pragma unroll
            for (int i = 0; i < JP / 2; ++i) {
              if (k0 + 4 * i <= M) *(float2*)(base + (to + 2 * i * row)) = make_float2(C[i].x, -D[i].x);
              if (k0 + 4 * i + 2 <= M) *(float2*)(base + (to + (2 * i + 1) * row)) = make_float2(C[i].y, -D[i].y);
            }
          }
        } else if (KIND == kFixInv) {
#pragma unroll
          for (int i = 0; i < JP / 2; ++i) {          // rows k, N - k
            const float2 y0 = make_float2(C[i].x + D[i].x, C[i].y + D[i].y), y1 = make_float2(C[i].x - D[i].x, C[i].y - D[i].y);
            C[i] = y0; D[i] = y1;
          }
          if (P.s == 1) {
            if (P.gelu) {
#pragma unroll
              for (int i = 0; i < JP / 2; ++i) { gelu_fast_pair(C[i].x, C[i].y); gelu_fast_pair(D[i].x, D[i].y); }
            }
            char* base = (char*)((IO*)P.out + (size_t)(P.plane0 + first) * P.OH * P.OW);
            const int oy = k0 - P.po, om = N - k0 - P.po, row = P.OW * (int)sizeof(IO);
            const int to = ((pl - first) * P.OH * P.OW + at - P.po) * (int)sizeof(IO);
            if (valid) {
#pragma unroll
              for (int i = 0; i < JP; ++i) {
                const int k = k0 + 2 * i;
                if (k <= M && (unsigned)(oy + 2 * i) < (unsigned)P.OH)
                  st_io<IO>(base + (uint32_t)(to + (oy + 2 * i) * row), 0, i & 1 ? C[i / 2].y : C[i / 2].x);
                if (k > 0 && k < M && (unsigned)(om - 2 * i) < (unsigned)P.OH)
                  st_io<IO>(base + (uint32_t)(to + (om - 2 * i) * row), 0, i & 1 ? D[i / 2].y : D[i / 2].x);
              }
            }
          } else if (valid) {
            char* base = (char*)(P.r + (size_t)first * N * P.wp);
            const uint32_t row = (uint32_t)P.wp * 4, to = (uint32_t)((pl - first) * N * P.wp + at) * 4;
#pragma unroll
            for (int i = 0; i < JP; ++i) {
              const int k = k0 + 2 * i;
              if (k <= M) *(float*)(base + (to + (uint32_t)k * row)) = i & 1 ? C[i / 2].y : C[i / 2].x;
              if (k > 0 && k < M) *(float*)(base + (to + (uint32_t)(N - k) * row)) = i & 1 ? D[i / 2].y : D[i / 2].x;
            }
          }
        } else {
          // the row's other part lives in the neighbouring lane; this one finishes frequency k, that one N - k
          float2* to = (float2*)smem + (line >> 1);
          const float sg = P.conj ? -1.f : 1.f;
#pragma unroll
          for (int i = 0; i < JP; ++i) {
            const int k = k0 + 2 * i;
            const float c = i & 1 ? C[i / 2].y : C[i / 2].x, s = i & 1 ? D[i / 2].y : D[i / 2].x;
            const float o = __shfl_xor_sync(0xffffffffu, c, 1), p = __shfl_xor_sync(0xffffffffu, s, 1);
            const float a = c + p, b = o - s;
            float2 z = mirror ? make_float2(b, a) : make_float2(a, b);
            if (pass == 0) {
              const float2 g = make_float2(gt[i].x, sg * gt[i].y);
              z = make_float2(fmaf(-z.y, g.y, z.x * g.x), -fmaf(z.x, g.y, z.y * g.x));
            }
            if (k <= M && !(mirror && (k == 0 || k == M))) {
              to[(mirror ? N - k : k) * kFixPitch] = z;
            }
          }
        }
      }
    }
    if (KIND == kFixRows) {
      __syncthreads();
      fix_exchange(P, smem, tile, tile + gridDim.x, tiles);
    }
  }
  fx_before_sync();
  __syncthreads();
  if (!ok && P.status) atomicExch(P.status, 5);
  if (warp == 0) fx_free(tm);
}

}  // namespace rp
}  // namespace cvb
