// The channel-mixing parts of ConverseBlock on tcgen05, one kernel for each side of the Converse2D operator:
//   PRE :  out = GELU( W1 . LN(x) + b1 )                                   64 -> 128 channels
//   POST:  x1 = x + a1 (W2 . t + b2);  out = x1 + a2 (W4 . GELU( W3 . LN(x1) + b3 ) + b4)    t: 128, x, out: 64
// (models/util_converse.py:278-293, 321-322).  A thread owns a pixel from its loads to its stores: LayerNorm, GELU,
// residuals and the operands of all three contractions of POST stay inside one thread and its lane of tensor memory,
// so the 128-channel hidden tensor and x1 never leave the SM.
//
// A block is two groups of 256 threads; each works on a 128-pixel tile of its own, so that one group's arithmetic
// covers the other's MMAs.  Two threads share a pixel, 32 channels each (sixteen warps on an SM: with one thread per
// pixel and eight warps 8 x 256 x 256 pixels of POST took 239 us); they meet only in LayerNorm and in the scale of t, through
// shared memory.  Per contraction: the thread splits its values into fp16 hi + lo and writes them to its lane of one of the
// group's two operand buffers (tcgen05.st, 64 channels at a time); after a barrier of the group one warp issues
// hi hi + hi lo + lo hi with the weights from shared memory and commits to the group's mbarrier; every thread then reads its
// half of its lane of the accumulator.  TMEM columns of group g at 256 g: accumulator [0,128), operands [128,192) and
// [192,256).  The weights, scaled, split and in operand layout, were packed once (block_pack_kernel) and arrive by one bulk
// copy.  Rows that are 16-byte aligned are copied to shared memory two phases and more ahead of their use, each warp its own
// 32 channels x 32 pixels; others are loaded pixel by pixel (any image size and alignment, fp32 or bf16).
//
// fp16 hi + lo keeps 22 bits of a value like TF32 hi + lo, with K = 16 an MMA instead of 8 and half the space, as long as the
// values lie high enough in fp16's range (cvb_mix.cuh states the bound): rows of weights, hidden channels and pixels are scaled
// by powers of two.  A LayerNorm's values stay below 8, each hidden channel below a bound that follows from its weights; t has
// any size that fp32 has, so a pixel takes its scale from its first 64 channels, and if the others are more than 32 times as
// large its sums so far are scaled down in tensor memory.
// With TF32 (twice as many MMAs, whose 46 cycles at least the two groups wait for together, and waits for one operand buffer)
// 8 x 256 x 256 pixels took 103 us PRE and 232 POST, with fp16 93 and 199, with the copies ahead 81 and 164; against fp64
// PRE's error went from 5.9e-7 to 3.6e-7, POST's from 1.0e-6 to 5.8e-7.
//
// What bounds it: bytes (PRE 3 C, POST 4 C channel planes: 61 and 82 us) and, in POST, a group's chain of five contractions
// with the arithmetic between them.  Registers spilled to local memory cost far more than their number suggests, because the
// shared memory leaves the L1 cache next to nothing (POST with 33 words spilled: 192 us).
// Every wait is bounded; after a time-out a thread stops working but keeps meeting the group's barriers.
#include "../../include/converse_b200.h"
#include "cvb_internal.h"
#include "cvb_mix.cuh"

namespace cvb {

// ---- packed weights: PRE | POST, each a multiple of 16 bytes: matrices as fp16 hi and lo (16 KB each), every row scaled by a
// power of two to below 2^14, then fp32 vectors.  The factors that undo the scales of a row and of its operand are in the
// vectors: 1 / (row scale x kNormScale) for what follows a LayerNorm (its values stay below 8), 1 / row scale for W2 and W4.  Every
// hidden value has a scale of its own (a bound of it follows from its row of W3 and its b3), which W4's columns undo before
// its rows are scaled: with one scale for all 128, a row of W3 2^20 times the others left these only their hi halves' bits.
// t is scaled pixel by pixel.
constexpr float kNormScale = 1024.f;
constexpr int kPreFloats = kW + 2 * kBlkM;                      // W1; b1, undo1
constexpr int kPostFloats = 3 * kW + 6 * kBlkC + 2 * kBlkM + kBlkM / 2; // W2, W3, W4; b2, a1, b4, a2, undo2, undo4; b3, undo3;
                                                                // hidden scales (powers of two, as bf16)
enum { kB2 = 0, kA1 = kBlkC, kB4 = 2 * kBlkC, kA2 = 3 * kBlkC, kUndo2 = 4 * kBlkC, kUndo4 = 5 * kBlkC, kB3 = 6 * kBlkC,
       kUndo3 = 6 * kBlkC + kBlkM, kHidden = 6 * kBlkC + 2 * kBlkM };
size_t block_pack_bytes() { return (size_t)(kPreFloats + kPostFloats) * sizeof(float); }

struct PackParams {
  const float *ln1_w, *ln1_b, *w1, *b1, *w2, *b2, *a1, *ln2_w, *ln2_b, *w3, *b3, *w4, *b4, *a2;
  float* out;
};

// the power of two that takes m to [2^13, 2^14), at most 2^most (1 for zero, infinities and NaN)
__device__ __forceinline__ float to_2_14(float m, int most) {
  const int e = (int)(__float_as_uint(m) >> 23);
  if (e == 0 || e >= 255) return 1.f;
  const int f = 127 + 13 + 127 - e;
  return __uint_as_float((uint32_t)(f < 1 ? 1 : f > 127 + most ? 127 + most : f) << 23);
}

// grid: 4 matrices x 16 slices.  The LayerNorm affine is folded into the weights that follow it.
__global__ void __launch_bounds__(256) block_pack_kernel(const PackParams P) {
  __shared__ float hidden[kBlkM];
  const int which = blockIdx.x >> 4, slice = blockIdx.x & 15, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* post = P.out + kPreFloats;
  const float* w = which == 0 ? P.w1 : which == 1 ? P.w2 : which == 2 ? P.w3 : P.w4;
  const float* g = which == 0 ? P.ln1_w : which == 2 ? P.ln2_w : nullptr;
  const int N = which == 0 || which == 2 ? kBlkM : kBlkC, K = kW / N;
  __half* hi = (__half*)(which == 0 ? P.out : post + (which - 1) * kW);
  float* vec = which == 0 ? P.out + kW : post + 3 * kW;
  const float* bias = which == 0 ? P.b1 : which == 1 ? P.b2 : which == 2 ? P.b3 : P.b4;
  const float* beta = which == 0 ? P.ln1_b : which == 2 ? P.ln2_b : nullptr;
  // the hidden values' bounds: |W3 . v + b3'| <= 8 |W3 row| + |b3'| for a normalised v of 64 values
  if (which == 3 || (which == 2 && slice == 0)) {
    for (int n = warp; n < kBlkM; n += 8) {
      float q = 0.f, d = 0.f;
      for (int k = lane; k < kBlkC; k += 32) {
        const float a = P.w3[n * kBlkC + k];
        q = fmaf(a * P.ln2_w[k], a * P.ln2_w[k], q);
        d = fmaf(a, P.ln2_b[k], d);
      }
      for (int o = 16; o; o >>= 1) { q += __shfl_xor_sync(0xffffffffu, q, o); d += __shfl_xor_sync(0xffffffffu, d, o); }
      const float most = 8.f * sqrtf(q) + fabsf(d + P.b3[n]);
      if (lane == 0) hidden[n] = most > 0.f ? to_2_14(1.001f * most, 100) : 0x1p100f;      // (1.001: sums are rounded; 2^100: W4's columns stay normal)
    }
    __syncthreads();
    if (which == 2 && threadIdx.x < kBlkM) {       // a thread's 32 of each 64 channels lie behind its other vectors' channels
      const int n = threadIdx.x;
      ((__nv_bfloat16*)(vec + kHidden))[(n & 32) * 2 + (n >> 6) * 32 + (n & 31)] = __float2bfloat16(hidden[n]);
    }
  }
  auto weight = [&](int n, int k) {
    const float a = w[n * K + k];
    return g ? a * g[k] : which == 3 ? a / hidden[k] : a;
  };
  const int rows = N / 16;
  for (int r = warp; r < rows; r += 8) {
    const int n = slice * rows + r;
    float m = 0.f, d = 0.f;
    for (int k = lane; k < K; k += 32) {
      m = fmaxf(m, fabsf(weight(n, k)));
      if (beta) d = fmaf(w[n * K + k], beta[k], d);
    }
    for (int o = 16; o; o >>= 1) { m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o)); d += __shfl_xor_sync(0xffffffffu, d, o); }
    const float f = to_2_14(m, 126);
    for (int k = lane; k < K; k += 32) {
      const float a = weight(n, k) * f;
      const __half h = __float2half_rn(a);
      hi[pack_index16(N, n, k)] = h;
      hi[kW + pack_index16(N, n, k)] = __float2half_rn(a - __half2float(h));
    }
    if (lane) continue;
    const float b = bias[n] + d;
    if (which == 0) { vec[n] = b; vec[kBlkM + n] = 1.f / f / kNormScale; }
    if (which == 1) { vec[kB2 + n] = b; vec[kUndo2 + n] = 1.f / f; vec[kA1 + n] = P.a1 ? P.a1[n] : 1.f; }
    if (which == 2) { vec[kB3 + n] = b; vec[kUndo3 + n] = 1.f / f / kNormScale; }
    if (which == 3) { vec[kB4 + n] = b; vec[kUndo4 + n] = 1.f / f; vec[kA2 + n] = P.a2 ? P.a2[n] : 1.f; }
  }
}

int launch_block_pack(const float* ln1_w, const float* ln1_b, const float* w1, const float* b1, const float* w2,
                      const float* b2, const float* a1, const float* ln2_w, const float* ln2_b, const float* w3,
                      const float* b3, const float* w4, const float* b4, const float* a2, void* pack, cudaStream_t st) {
  const PackParams P = {ln1_w, ln1_b, w1, b1, w2, b2, a1, ln2_w, ln2_b, w3, b3, w4, b4, a2, (float*)pack};
  block_pack_kernel<<<64, 256, 0, st>>>(P);
  CVB_CUDA(cudaGetLastError());
  return CVB_OK;
}

struct MixParams {
  const void* x;
  const void* t;
  void* out;
  const float* pack;
  float eps;
  int HW;
  long long npix;
  int* status;
  float *z, *x1;        // TRAIN: (B,128,HW), (B,64,HW)
};

// Shared memory behind the weights: every warp has two slots for 32 channels of its 32 pixels
constexpr int kSlot = 32 * 32 * 4, kRing = 16 * 2 * kSlot;

__device__ __forceinline__ void mix_copy(void* dst, const void* src, bool in) {       // zeros where `in` is false
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}

// TRAIN (fp32): also keeps what the gradients need -- PRE the hidden layer before its GELU (z), POST x1 and the hidden
// layer before its GELU -- and POST takes t before ITS GELU.  COPIES: rows are 16-byte aligned and reach shared memory by
// asynchronous copies ahead of their use.
template <bool POST, typename IO, bool TRAIN, bool COPIES>
__global__ void __launch_bounds__(kMixThreads, 1) block_mix_kernel(const __grid_constant__ MixParams P) {
  extern __shared__ __align__(128) float msm[];
  pdl_start();
  constexpr int kFloats = POST ? kPostFloats : kPreFloats;
  float* wts = msm;
  const float* vec = wts + (POST ? 3 : 1) * kW;     // (see block_pack_kernel)
  unsigned char* ring = (unsigned char*)(msm + kFloats);
  uint64_t* bars = (uint64_t*)(ring + kRing);       // MMA of group 0, 1; weights; first half of t of group 0, 1
  uint32_t* holder = (uint32_t*)(bars + 5);
  const int tid = threadIdx.x, warp = (int)tc::from_first(tid >> 5), ln = tid & 31, g = warp >> 3, m = tid & 127, hf = (warp >> 2) & 1;
  const bool lead = (warp & 7) == 0;               // the warp that issues the group's MMAs
  if (tid == 0) {
    for (int i = 0; i < 5; ++i) mbar_init(&bars[i], 1);
    mbar_fence_init();
    mbar_expect_tx(&bars[2], kFloats * 4);
    bulk_g2s(wts, P.pack + (POST ? kPreFloats : 0), kFloats * 4, &bars[2]);
  }
  if (warp == 0) tc::tmem_alloc(holder, 512);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tc::from_first(*holder) + 256u * (uint32_t)g;
  const uint32_t lane = tmem + ((uint32_t)((warp & 3) * 32) << 16) + 32u * (uint32_t)hf;   // 32 columns a thread
  const uint32_t op = lane + 128u - 16u * (uint32_t)hf;        // its 16 columns of the first operand buffer, the second 64 on
  uint64_t* done = &bars[g];
  uint32_t uses = 0, tiles = 0;                     // commits of this group so far, tiles
  bool ok = true;

  const long long ntiles = (P.npix + 127) / 128, step = 2ll * gridDim.x;
  const int HW = P.HW;
  constexpr int Cin = POST ? kBlkM : kBlkC, Cout = POST ? kBlkC : kBlkM;
  const IO* const in = (const IO*)(POST ? P.t : P.x) + (size_t)(32 * hf) * HW;      // this warp's channels of the first item
  // a pixel of a tile: image, position in it
  struct Place { bool valid; int img, pos; };
  auto place = [&](long long tile, int at) {
    const long long pix = tile * 128 + at;
    Place q;
    q.valid = pix < P.npix;
    q.img = !q.valid ? 0 : P.npix <= 0xffffffffll ? (int)((uint32_t)pix / (uint32_t)HW) : (int)(pix / HW);
    q.pos = q.valid ? (int)(pix - (long long)q.img * HW) : 0;
    return q;
  };
  auto commit_wait = [&]() {                        // the group's last MMAs have finished
    if (ok) ok = mbar_wait_bounded(done, uses & 1u, kWaitLimit);
    uses += 1;
    tc::fence_after_sync();
  };
  auto publish = [&]() {                            // operand columns written, accumulator read, by the whole group
    tc::fence_before_sync();
    mix_bar(g);
    tc::fence_after_sync();
  };
  // ---- the way of the input: items of 32 channels x 32 pixels, a warp's own, in the order they are needed (POST: t, t, x of
  // a tile), two slots by turns.  An item is asked for when the one before last has been used up, two phases or more before
  // its use; single 4-byte loads into registers, a phase ahead, had the warps wait for their load queue two fifths of the
  // time.  Rows that are not 16-byte aligned keep those: 4-byte copies are slower (2 x 111 x 167 pixels: 23.3 us against 18.5).
  constexpr int PX = 16 / (int)sizeof(IO), CH = 32 / PX, RS = 32 / CH;      // pixels of a copy, copies of a row, rows a step
  const int first_px = (m & ~31) + ln % CH * PX;
  uint32_t item = 0;                                // items used so far
  auto slot = [&](int w, uint32_t i) { return ring + (w * 2 + (int)(i & 1u)) * kSlot; };
  auto ask = [&](uint32_t i, const IO* from, int channels, const Place& q) {
    const int r = ln / CH;
    unsigned char* dst = slot(warp, i) + r * 32 * (int)sizeof(IO) + ln % CH * 16;
    const IO* src = q.valid ? from + ((size_t)q.img * channels + r) * HW + q.pos : from;
    const size_t rows = q.valid ? (size_t)RS * HW : 0;
#pragma unroll
    for (int c = 0; c < 32; c += RS, src += rows) mix_copy(dst + c * 32 * (int)sizeof(IO), src, q.valid);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // the next item's values of this thread's pixel (without copies: they are in v already)
  auto take = [&](float (&v)[32]) {
    if (!COPIES) return;
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    const IO* p = (const IO*)slot(warp, item) + ln;
#pragma unroll
    for (int c = 0; c < 32; ++c) v[c] = ld_io<IO>(p, (size_t)(c * 32));
    __syncwarp();
  };
  // a cell of the slot just used up, and the one of the other thread of the pixel
  auto mine = [&]() { return (float2*)slot(warp, item) + ln; };
  auto other = [&]() { return (const float2*)slot(warp ^ 4, item) + ln; };

  long long tile = blockIdx.x + (long long)g * gridDim.x;
  Place here = place(tile, m);
  float v[32];
  if (!COPIES) {
    mix_load<IO>(v, in + (size_t)here.img * Cin * HW + here.pos, HW, here.valid);
  } else {
    ask(0, in, Cin, place(tile, first_px));
    ask(1, in + (POST ? (size_t)64 * HW : 0), Cin, place(POST ? tile : tile + step, first_px));
  }
  if (ok) ok = mbar_wait_bounded(&bars[2], 0, kWaitLimit);   // weights
  for (; tile < ntiles; tile += step) {
    const bool valid = here.valid;
    IO* op_out = (IO*)P.out + ((size_t)here.img * Cout + (POST ? 32 : 64) * hf) * HW + here.pos;
    if constexpr (!POST) {
      take(v);
      mix_norm(v, P.eps, mine(), other(), g, kNormScale);
      mix_stage16(op, v);
      publish();
      if (lead) {
        const uint32_t e = tc::elect_one() & (ok ? 1u : 0u);
        mix_mma16<128>(tmem, tmem + 128u, (const __half*)wts, 0, false, e);
        if (e) tc::mma_commit(done);
      }
      if (!COPIES) {
        const Place q = place(tile + step, m);
        mix_load<IO>(v, in + (size_t)q.img * Cin * HW + q.pos, HW, q.valid);
      } else {
        ask(item + 2, in, Cin, place(tile + 2 * step, first_px));
      }
      item += 1;
      commit_wait();
#pragma unroll 1
      for (int c0 = 0; c0 < 64; c0 += 32) {         // 64 of the 128 output channels
        float a[32];
        tc::tmem_ld32(lane + (uint32_t)(32 * hf + c0), a);
        if (valid && ok) {
#ifdef __CUDA_ARCH__
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            const float2 b = *(const float2*)(vec + 64 * hf + c0 + j), u = *(const float2*)(vec + kBlkM + 64 * hf + c0 + j);
            const float za = fmaf(a[j], u.x, b.x), zb = fmaf(a[j + 1], u.y, b.y);
            const float2 o = gelu_fast2(za, zb);
            if (TRAIN) {
              float* zp = P.z + (op_out - (IO*)P.out);
              zp[(size_t)(c0 + j) * HW] = za;
              zp[(size_t)(c0 + j + 1) * HW] = zb;
            }
            st_io<IO>(op_out, (size_t)(c0 + j) * HW, o.x);
            st_io<IO>(op_out, (size_t)(c0 + j + 1) * HW, o.y);
          }
#endif
        }
      }
    } else {
      const __half *w2 = (const __half*)wts, *w3 = w2 + 2 * kW, *w4 = w3 + 2 * kW;
      const float* vh = vec + 32 * hf;              // this thread's channels of the vectors
      float x1[32];
      if (!COPIES) mix_load<IO>(x1, (const IO*)P.x + ((size_t)here.img * kBlkC + 32 * hf) * HW + here.pos, HW, valid);
      float undo = 1.f;                             // of the scale of t
      int top = 0;                                  //   and its exponent
      // five operands of 64 channels: t (two halves), LN(x1), GELU (two halves), in two buffers by turns.  One copy of the
      // staging code: the whole kernel has to stay in the instruction cache.
#pragma unroll 1
      for (int ph = 0; ph < 5; ++ph) {
        if (ph == 2) {                              // x1 = x + a1 (W2 . t + b2)
          if (COPIES) take(v);
          commit_wait();
          float a[32];
          tc::tmem_ld32(lane, a);
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            // (both factors are powers of two: their product first, or a sum times one of them may overflow alone)
            x1[j] = fmaf(vh[kA1 + j], fmaf(a[j], vh[kUndo2 + j] * undo, vh[kB2 + j]), COPIES ? v[j] : x1[j]);
            v[j] = x1[j];
            if (TRAIN && valid) P.x1[(op_out - (IO*)P.out) + (size_t)j * HW] = x1[j];
          }
          mix_norm(v, P.eps, mine(), other(), g, kNormScale);
        } else if (ph >= 3) {                       // GELU of 32 of 64 hidden channels
          const int h0 = 64 * (ph - 3);
          if (ph == 3) commit_wait();
          float a[32];
          tc::tmem_ld32(lane + (uint32_t)h0, a);
#ifdef __CUDA_ARCH__
          const uint32_t* hs = (const uint32_t*)(vh + kHidden) + h0 / 4;
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            const float2 b = *(const float2*)(vh + kB3 + h0 + j), u = *(const float2*)(vh + kUndo3 + h0 + j);
            const float za = fmaf(a[j], u.x, b.x), zb = fmaf(a[j + 1], u.y, b.y);
            const float2 o = gelu_fast2(za, zb);
            if (TRAIN && valid) {
              float* zp = P.z + ((size_t)here.img * kBlkM + h0 + 32 * hf) * HW + here.pos;
              zp[(size_t)j * HW] = za;
              zp[(size_t)(j + 1) * HW] = zb;
            }
            v[j] = o.x * __uint_as_float(hs[j / 2] << 16); v[j + 1] = o.y * __uint_as_float(hs[j / 2] & 0xffff0000u);
          }
#endif
        } else {                                    // 64 channels of t
          take(v);
#ifdef __CUDA_ARCH__
          if (TRAIN) {
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
              const float2 o = gelu_fast2(v[j], v[j + 1]);
              v[j] = o.x; v[j + 1] = o.y;
            }
          }
#endif
          // the pixel's largest magnitude goes to [2^10, 2^11): the other half may be 32 times as large
          float most = 0.f;
#pragma unroll
          for (int j = 0; j < 32; ++j) most = fmaxf(most, fabsf(v[j]));
          mine()->x = most;
          mix_bar(g);
          const int e = min(max((int)(__float_as_uint(fmaxf(most, other()->x)) >> 23), 11), 254);
          if (ph == 0) {
            top = e;
          } else if (__any_sync(0xffffffffu, e > top + 4)) {       // it is larger still: the sums so far are scaled down
            if (ok) ok = mbar_wait_bounded(&bars[3 + g], tiles & 1u, kWaitLimit);
            tc::fence_after_sync();
            const int by = e > top + 4 ? e - top : 0;
            const float f = by > 126 ? 0.f : __uint_as_float((uint32_t)(127 - by) << 23);
            top += by;
            float a[32];
            tc::tmem_ld32(lane, a);
            float b0[16], b1[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) { b0[j] = a[j] * f; b1[j] = a[16 + j] * f; }
            mix_st16(lane, b0);
            mix_st16(lane + 16u, b1);
            tc::tmem_wait_st();
          }
          const float s = __uint_as_float((uint32_t)min(264 - top, 254) << 23);       // 2^(10 - exponent)
          undo = 1.f / s;
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] *= s;
        }
        const uint32_t buf = 64u * (uint32_t)(ph & 1);
        mix_stage16(op + buf, v);
        publish();                                  // (the accumulator's first 64 columns have been read by ph = 3)
        if (lead) {
          const uint32_t e = tc::elect_one() & (ok ? 1u : 0u);
          if (ph == 2) mix_mma16<128>(tmem, tmem + 128u + buf, w3, 0, false, e);
          else mix_mma16<64>(tmem, tmem + 128u + buf, ph < 2 ? w2 : w4, ph == 1 || ph == 4 ? 64 : 0, ph == 1 || ph == 4, e);
          if (e && ph != 3) tc::mma_commit(ph == 0 ? &bars[3 + g] : done);
        }
        // what comes after next: x after the first half of t, then the next tile's two halves
        if (!COPIES) {
          if (ph == 0 || ph == 4) {
            const Place q = ph == 4 ? place(tile + step, m) : here;
            mix_load<IO>(v, in + (ph == 0 ? (size_t)64 * HW : 0) + (size_t)q.img * Cin * HW + q.pos, HW, q.valid);
          }
        } else if (ph < 3) {
          ask(item + 2, ph == 0 ? (const IO*)P.x + (size_t)(32 * hf) * HW : in + (ph == 2 ? (size_t)64 * HW : 0),
              ph == 0 ? kBlkC : kBlkM, place(ph == 0 ? tile : tile + step, first_px));
        }
        if (ph < 3) item += 1;
      }
      tiles += 1;
      commit_wait();
      float a[32];
      tc::tmem_ld32(lane, a);
      if (valid && ok) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          st_io<IO>(op_out, (size_t)j * HW, fmaf(vh[kA2 + j], fmaf(a[j], vh[kUndo4 + j], vh[kB4 + j]), x1[j]));
      }
    }
    here = place(tile + step, m);
  }
  if (!ok && P.status) atomicExch(P.status, 3);
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(*holder, 512);
}

template <bool POST, typename IO, bool TRAIN, bool COPIES>
static int launch_one(const MixParams& P, int sms, cudaStream_t st) {
  const size_t smem = (size_t)(POST ? kPostFloats : kPreFloats) * sizeof(float) + kRing + 5 * sizeof(uint64_t) + 8;
  const int rc = allow_smem(block_mix_kernel<POST, IO, TRAIN, COPIES>, smem);
  if (rc != CVB_OK) return rc;
  const long long ntiles = (P.npix + 127) / 128;
  const int grid = (int)(ntiles < sms ? ntiles : sms);     // one block per SM; tiles go round the blocks first
  return launch_chained(block_mix_kernel<POST, IO, TRAIN, COPIES>, dim3(grid), kMixThreads, smem, st, P);
}
template <bool POST, typename IO, bool TRAIN = false>
static int launch_mix(const MixParams& P, int sms, cudaStream_t st) {
  const size_t at = (size_t)P.x | (size_t)(POST ? P.t : P.x) | (size_t)P.HW * sizeof(IO);
  return at % 16 == 0 ? launch_one<POST, IO, TRAIN, true>(P, sms, st) : launch_one<POST, IO, TRAIN, false>(P, sms, st);
}

int launch_block_mix(bool post, const void* x, const void* t, void* out, const void* pack, float eps, int B, int HW,
                     int io_dtype, int sms, int* status, cudaStream_t st) {
  MixParams P;
  P.x = x; P.t = t; P.out = out; P.pack = (const float*)pack; P.eps = eps;
  P.HW = HW; P.npix = (long long)B * HW; P.status = status; P.z = nullptr; P.x1 = nullptr;
  if (post) return io_dtype == CVB_F32 ? launch_mix<true, float>(P, sms, st) : launch_mix<true, __nv_bfloat16>(P, sms, st);
  return io_dtype == CVB_F32 ? launch_mix<false, float>(P, sms, st) : launch_mix<false, __nv_bfloat16>(P, sms, st);
}

int launch_block_mix_train(bool post, const float* x, const float* t, float* out, float* z, float* x1, const void* pack,
                           float eps, int B, int HW, int sms, int* status, cudaStream_t st) {
  MixParams P;
  P.x = x; P.t = t; P.out = out; P.pack = (const float*)pack; P.eps = eps;
  P.HW = HW; P.npix = (long long)B * HW; P.status = status; P.z = z; P.x1 = x1;
  return post ? launch_mix<true, float, true>(P, sms, st) : launch_mix<false, float, true>(P, sms, st);
}

}  // namespace cvb
