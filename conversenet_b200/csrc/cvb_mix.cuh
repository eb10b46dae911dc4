// Building blocks of the ConverseBlock kernels on tcgen05 (k_block_mlp.cu: forward, k_block_train.cu: gradients): operand
// staging in tensor memory, the split MMAs, LayerNorm over the two threads of a pixel.
#pragma once
#include "cvb_block.cuh"
#include "cvb_tc.cuh"
#include <cuda_fp16.h>

namespace cvb {

constexpr int kW = kBlkC * kBlkM;                               // values of one weight matrix

// float index of element (n, k) of an operand with N rows (K-major core matrices, no swizzle)
__host__ __device__ constexpr int pack_index(int N, int n, int k) {
  return (n >> 3) * 32 + (n & 7) * 4 + (k & 3) + ((k >> 2) & 1) * (N / 8) * 32 + (k >> 3) * (N / 8) * 64;
}

constexpr int kMixThreads = 512;
constexpr uint32_t kOpHi = 128, kOpLo = 192;

// sixteen consecutive columns of this thread's TMEM lane
__device__ __forceinline__ void mix_st16(uint32_t taddr, const float (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])),
      "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])), "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])),
      "r"(__float_as_uint(v[8])), "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])), "r"(__float_as_uint(v[11])),
      "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])), "r"(__float_as_uint(v[14])), "r"(__float_as_uint(v[15]))
      : "memory");
}
// this thread's 32 of 64 channel values -> operand columns (lane: its half's first column of the accumulator)
__device__ __forceinline__ void mix_stage(uint32_t lane, const float (&v)[32]) {
#pragma unroll
  for (int c0 = 0; c0 < 32; c0 += 16) {
    float hi[16], lo[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) tc::split_tf32(v[c0 + e], hi[e], lo[e]);
    mix_st16(lane + kOpHi + (uint32_t)c0, hi);
    mix_st16(lane + kOpLo + (uint32_t)c0, lo);
  }
  tc::tmem_wait_st();
}
// D (+)= A[64 channels in the operand columns] . B, B = N rows, K columns k0 .. k0 + 63 of a packed matrix
template <int N>
__device__ __forceinline__ void mix_mma(uint32_t tmem, const float* b_hi, int k0, bool accumulate, uint32_t elected) {
  constexpr uint32_t idesc = tc::idesc_tf32(128, N, false, false);
  constexpr int LBO = (N / 8) * 128, KSTEP = 2 * LBO;
#pragma unroll
  for (int ks = 0; ks < 8; ++ks) {
    const uint64_t bh = tc::smem_desc((const char*)b_hi + (k0 / 8 + ks) * KSTEP, LBO, 128);
    const uint64_t bl = tc::smem_desc((const char*)(b_hi + kW) + (k0 / 8 + ks) * KSTEP, LBO, 128);
    tc::mma_tf32_ta(tmem, tmem + kOpHi + ks * 8, bh, idesc, (accumulate || ks > 0) ? 1u : 0u, elected);
    tc::mma_tf32_ta(tmem, tmem + kOpHi + ks * 8, bl, idesc, 1u, elected);
    tc::mma_tf32_ta(tmem, tmem + kOpLo + ks * 8, bh, idesc, 1u, elected);
  }
}

// ---- the forward's operands: fp16 hi + lo, at twice the rate of TF32 hi + lo and half the space.  The values of a row are
// scaled by a power of two, the largest to below 2^14.  A value then keeps 22 bits, as TF32 hi + lo does, down to 2^-3 (its lo
// half is a normal number), and an absolute error of 2^-25 below: 2^-39 of the bound of a row of weights or of a hidden channel,
// 2^-38 of a LayerNorm's bound of 8 (which a pixel whose channels differ by far less than eps comes nowhere near), 2^-35 of a
// pixel's largest value of t.  TF32 would keep 22 bits of values smaller still; a sum in fp32 would not show them
// unless the other operand makes up for it.
// half index of element (n, k) of an operand with N rows (K-major core matrices of 8 x 8, no swizzle)
__host__ __device__ constexpr int pack_index16(int N, int n, int k) {
  return (n >> 3) * 64 + (n & 7) * 8 + (k & 7) + ((k >> 3) & 1) * (N / 8) * 64 + (k >> 4) * (N / 8) * 128;
}
// this thread's 32 of 64 channel values -> operand columns (two channels a column: hi 32 columns, lo 32); `op`: this
// thread's lane, its half's first column
__device__ __forceinline__ void mix_stage16(uint32_t op, const float (&v)[32]) {
  float hi[16], lo[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const __half2 h = __floats2half2_rn(v[2 * e], v[2 * e + 1]);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(v[2 * e] - f.x, v[2 * e + 1] - f.y);
    hi[e] = __uint_as_float(*(const uint32_t*)&h);
    lo[e] = __uint_as_float(*(const uint32_t*)&l);
  }
  mix_st16(op, hi);
  mix_st16(op + 32u, lo);
  tc::tmem_wait_st();
}
// D (+)= A[64 channels in the operand columns from `op` on] . B, B = N rows, K columns k0 .. k0 + 63 of a matrix packed with
// pack_index16, lo behind hi; a whole warp
template <int N>
__device__ __forceinline__ void mix_mma16(uint32_t tmem, uint32_t op, const __half* b, int k0, bool accumulate, uint32_t elected) {
  constexpr uint32_t idesc = (1u << 4) | ((uint32_t)(N >> 3) << 17) | (8u << 24);     // fp16 operands, fp32 sums, M = 128
  constexpr int LBO = (N / 8) * 128, KSTEP = 2 * LBO;
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) {
    const uint64_t bh = tc::smem_desc((const char*)b + (k0 / 16 + ks) * KSTEP, LBO, 128);
    const uint64_t bl = tc::smem_desc((const char*)(b + kW) + (k0 / 16 + ks) * KSTEP, LBO, 128);
    tc::mma_f16_ta(tmem, op + ks * 8, bh, idesc, (accumulate || ks > 0) ? 1u : 0u, elected);
    tc::mma_f16_ta(tmem, op + ks * 8, bl, idesc, 1u, elected);
    tc::mma_f16_ta(tmem, op + 32 + ks * 8, bh, idesc, 1u, elected);
  }
}
template <typename IO>
__device__ __forceinline__ void mix_load(float (&v)[32], const IO* p, int HW, bool valid) {
#pragma unroll
  for (int c = 0; c < 32; ++c) v[c] = valid ? ld_io<IO>(p, (size_t)c * HW) : 0.f;
}
__device__ __forceinline__ void mix_bar(int g) {
  if (g == 0) asm volatile("bar.sync 1, 256;" ::: "memory");
  else asm volatile("bar.sync 2, 256;" ::: "memory");
}
// centre and scale a pixel's 64 values (and times `scale`), 32 of them here (the affine part is in the weights).  `mine`, `other`: this and
// the partner thread's cell for (mean, sum of squared deviations) of a half; the two combine to the whole's.
__device__ __forceinline__ float mix_norm(float (&v)[32], float eps, float2* mine, const float2* other, int g, float scale = 1.f) {
  float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
  for (int c = 0; c < 32; c += 4) { s0 += v[c]; s1 += v[c + 1]; s2 += v[c + 2]; s3 += v[c + 3]; }
  const float m0 = ((s0 + s1) + (s2 + s3)) * (1.0f / 32);
  s0 = s1 = s2 = s3 = 0.f;
#pragma unroll
  for (int c = 0; c < 32; c += 4) {
    const float a = v[c] - m0, b = v[c + 1] - m0, d = v[c + 2] - m0, e = v[c + 3] - m0;
    s0 = fmaf(a, a, s0); s1 = fmaf(b, b, s1); s2 = fmaf(d, d, s2); s3 = fmaf(e, e, s3);
  }
  const float q0 = (s0 + s1) + (s2 + s3);
  *mine = make_float2(m0, q0);
  mix_bar(g);
  const float2 o = *other;
  const float d = m0 - o.x, mean = 0.5f * (m0 + o.x);
  const float rstd = 1.0f / sqrtf(fmaf(16.f * d, d, q0 + o.y) * (1.0f / 64) + eps);
#pragma unroll
  for (int c = 0; c < 32; ++c) v[c] = (v[c] - mean) * (rstd * scale);
  return rstd;
}

}  // namespace cvb
