// The channel-mixing parts of ConverseBlock on tcgen05, one kernel for each side of the Converse2D operator:
//   PRE :  out = GELU( W1 . LN(x) + b1 )                                   64 -> 128 channels
//   POST:  x1 = x + a1 (W2 . t + b2);  out = x1 + a2 (W4 . GELU( W3 . LN(x1) + b3 ) + b4)    t: 128, x, out: 64
// (models/util_converse.py:278-293, 321-322).  A thread owns a pixel from its loads to its stores: LayerNorm, GELU,
// residuals and the operands of all three contractions of POST stay inside one thread and its lane of tensor memory,
// so the 128-channel hidden tensor and x1 never leave the SM.
//
// A block is two groups of 256 threads; each works on a 128-pixel tile of its own, so that one group's arithmetic
// covers the other's MMAs.  Two threads share a pixel, 32 channels each (sixteen warps on an SM: with one thread per
// pixel and eight warps 8 x 256 x 256 pixels of POST took 239 us); they meet only in LayerNorm, whose halves' means and
// squared deviations go through shared memory.  Per contraction: the thread splits its values into TF32 hi + lo and
// writes them to its lane of the group's operand columns (tcgen05.st, 64 channels at a time); after a barrier of the
// group one thread issues hi hi + hi lo + lo hi with the weights from shared memory and commits to the group's mbarrier;
// every thread then reads its half of its lane of the accumulator.  TMEM columns of group g at 256 g: accumulator
// [0,128), operand hi [128,192), lo [192,256).  The weights, split and in operand layout, were packed once
// (block_pack_kernel) and arrive by one bulk copy.  Pixels are addressed one by one (channel rows of any alignment, any
// image size, fp32 or bf16); the values of the next tile are requested while the current one computes.
//
// What bounds it: bytes (PRE 3 C, POST 4 C channel planes), the MMAs (24 of 128x128x8 a tile for PRE, 72 of which 48 of
// 128x64x8 for POST) and instruction issue (about 2400 and 4000 a warp and tile).  8 x 256 x 256 pixels, fp32: PRE and POST
// take 337 us, their 940 MB would take 144.  PRE has 62 % of its issue slots busy and DRAM at 38 %; POST 43 % and 26 %, the
// tensor pipe at 39 %, and waits for its 192 channel rows a tile: 202 KB of weights leave one block an SM and no ring.
// Every wait is bounded; after a time-out a thread stops working but keeps meeting the group's barriers.
#include "../../include/converse_b200.h"
#include "cvb_internal.h"
#include "cvb_mix.cuh"

namespace cvb {

// ---- packed weights: PRE | POST, each a multiple of 16 bytes
constexpr int kPreFloats = 2 * kW + kBlkM;                      // W1 hi, lo; b1
constexpr int kPostFloats = 6 * kW + 4 * kBlkC + kBlkM;         // W2, W3, W4 hi, lo; b2, a1, b4, a2; b3
size_t block_pack_bytes() { return (size_t)(kPreFloats + kPostFloats) * sizeof(float); }

struct PackParams {
  const float *ln1_w, *ln1_b, *w1, *b1, *w2, *b2, *a1, *ln2_w, *ln2_b, *w3, *b3, *w4, *b4, *a2;
  float* out;
};

// grid: 4 matrices x 16 slices.  The LayerNorm affine is folded into the weights that follow it.
__global__ void __launch_bounds__(256) block_pack_kernel(const PackParams P) {
  const int which = blockIdx.x >> 4, slice = blockIdx.x & 15;
  float* post = P.out + kPreFloats;
  const float* w = which == 0 ? P.w1 : which == 1 ? P.w2 : which == 2 ? P.w3 : P.w4;
  const float* g = which == 0 ? P.ln1_w : which == 2 ? P.ln2_w : nullptr;
  const int N = which == 0 || which == 2 ? kBlkM : kBlkC, K = kW / N;
  float* hi = which == 0 ? P.out : post + (which - 1) * 2 * kW;
  for (int i = slice * (kW / 16) + threadIdx.x; i < (slice + 1) * (kW / 16); i += 256) {
    const int n = i / K, k = i - n * K;
    float a, b;
    tc::split_tf32(g ? w[i] * g[k] : w[i], a, b);
    hi[pack_index(N, n, k)] = a;
    hi[kW + pack_index(N, n, k)] = b;
  }
  if (slice != 0) return;
  float* vec = post + 6 * kW;
  const float* bias = which == 0 ? P.b1 : which == 1 ? P.b2 : which == 2 ? P.b3 : P.b4;
  const float* beta = which == 0 ? P.ln1_b : which == 2 ? P.ln2_b : nullptr;
  float* dst = which == 0 ? P.out + 2 * kW : which == 1 ? vec : which == 2 ? vec + 4 * kBlkC : vec + 2 * kBlkC;
  for (int n = threadIdx.x; n < N; n += 256) {
    float s = bias[n];
    if (beta)
      for (int k = 0; k < K; ++k) s = fmaf(w[n * K + k], beta[k], s);
    dst[n] = s;
    if (which == 1) vec[kBlkC + n] = P.a1 ? P.a1[n] : 1.0f;
    if (which == 3) vec[3 * kBlkC + n] = P.a2 ? P.a2[n] : 1.0f;
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

// TRAIN (fp32): also keeps what the gradients need -- PRE the hidden layer before its GELU (z), POST x1 and the hidden
// layer before its GELU -- and POST takes t before ITS GELU.
template <bool POST, typename IO, bool TRAIN>
__global__ void __launch_bounds__(kMixThreads, 1) block_mix_kernel(const __grid_constant__ MixParams P) {
  extern __shared__ __align__(128) float msm[];
  pdl_start();
  constexpr int kFloats = POST ? kPostFloats : kPreFloats;
  float* wts = msm;
  const float* vec = wts + (POST ? 6 : 2) * kW;    // PRE: b1.  POST: b2, a1, b4, a2, b3
  uint64_t* bars = (uint64_t*)(msm + kFloats);      // MMA of group 0, 1; weights
  uint32_t* holder = (uint32_t*)(bars + 3);
  float2* halves = (float2*)(holder + 2);           // [group][half][pixel]
  const int tid = threadIdx.x, warp = tid >> 5, g = tid >> 8, m = tid & 127, hf = (tid >> 7) & 1;
  const bool lead = (tid & 255) == 0;
  float2* mine = halves + (g * 2 + hf) * 128 + m;
  const float2* other = halves + (g * 2 + (hf ^ 1)) * 128 + m;
  if (tid == 0) {
    for (int i = 0; i < 3; ++i) mbar_init(&bars[i], 1);
    mbar_fence_init();
    mbar_expect_tx(&bars[2], kFloats * 4);
    bulk_g2s(wts, P.pack + (POST ? kPreFloats : 0), kFloats * 4, &bars[2]);
  }
  if (warp == 0) tc::tmem_alloc(holder, 512);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *holder + 256u * (uint32_t)g;
  const uint32_t lane = tmem + ((uint32_t)((warp & 3) * 32) << 16) + 32u * (uint32_t)hf;   // 32 columns a thread
  uint64_t* done = &bars[g];
  uint32_t uses = 0;                                // commits of this group so far
  bool ok = true;

  const long long ntiles = (P.npix + 127) / 128, step = 2ll * gridDim.x;
  const int HW = P.HW;
  const int Cin = POST ? kBlkM : kBlkC, Cout = POST ? kBlkC : kBlkM;
  // this thread's pixel of a tile: image, position
  auto place = [&](long long tile, bool& valid, long long& img, int& pos) {
    const long long pix = tile * 128 + m;
    valid = pix < P.npix;
    img = valid ? pix / HW : 0;
    pos = valid ? (int)(pix - img * HW) : 0;
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

  long long tile = blockIdx.x + (long long)g * gridDim.x;
  bool valid = false;
  long long img = 0;
  int pos = 0;
  const size_t half_off = (size_t)(32 * hf) * HW;
  float v[32];
  if (tile < ntiles) {
    place(tile, valid, img, pos);
    mix_load<IO>(v, (const IO*)(POST ? P.t : P.x) + (size_t)img * Cin * HW + pos + half_off, HW, valid);
  }
  if (ok) ok = mbar_wait_bounded(&bars[2], 0, kWaitLimit);   // weights
  for (; tile < ntiles; tile += step) {
    const long long ntile = tile + step;
    bool nvalid = false;
    long long nimg = 0;
    int npos = 0;
    if (ntile < ntiles) place(ntile, nvalid, nimg, npos);
    const IO* next = (const IO*)(POST ? P.t : P.x) + (size_t)nimg * Cin * HW + npos + half_off;
    IO* op = (IO*)P.out + (size_t)img * Cout * HW + pos + (POST ? half_off : 2 * half_off);
    {
      // the tile after: rows of its first pixel in this warp
      const long long npix0 = ntile * 128 + (m & ~31);
      if (npix0 < P.npix) {
        const long long i0 = npix0 / HW;
        const size_t p0 = (size_t)(npix0 - i0 * HW) + half_off;
        const IO* q = (const IO*)(POST ? P.t : P.x) + (size_t)i0 * Cin * HW + p0;
        mix_prefetch<IO>(q, HW);
        if (POST) {
          mix_prefetch<IO>(q + (size_t)64 * HW, HW);
          mix_prefetch<IO>((const IO*)P.x + (size_t)i0 * kBlkC * HW + p0, HW);
        }
      }
    }
    if constexpr (!POST) {
      mix_norm(v, P.eps, mine, other, g);
      mix_stage(lane, v);
      publish();
      if (lead && ok) { mix_mma<128>(tmem, wts, 0, false); tc::mma_commit(done); }
      mix_load<IO>(v, next, HW, nvalid);
      commit_wait();
#pragma unroll 1
      for (int c0 = 0; c0 < 64; c0 += 32) {         // 64 of the 128 output channels
        float a[32];
        tc::tmem_ld32(lane + (uint32_t)(32 * hf + c0), a);
        if (valid && ok) {
#ifdef __CUDA_ARCH__
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            const float2 b = *(const float2*)(vec + 64 * hf + c0 + j);
            const float za = a[j] + b.x, zb = a[j + 1] + b.y;
            const float2 o = gelu_fast2(za, zb);
            if (TRAIN) {
              float* zp = P.z + (op - (IO*)P.out);
              zp[(size_t)(c0 + j) * HW] = za;
              zp[(size_t)(c0 + j + 1) * HW] = zb;
            }
            st_io<IO>(op, (size_t)(c0 + j) * HW, o.x);
            st_io<IO>(op, (size_t)(c0 + j + 1) * HW, o.y);
          }
#endif
        }
      }
    } else {
      const float *w2 = wts, *w3 = wts + 2 * kW, *w4 = wts + 4 * kW;
      const float* vh = vec + 32 * hf;              // this thread's channels of b2, a1, b4, a2
      float x1[32];
      mix_load<IO>(x1, (const IO*)P.x + (size_t)img * kBlkC * HW + pos + half_off, HW, valid);
      // five operands of 64 channels: t (two halves), LN(x1), GELU (two halves).  One copy of the staging code: the whole
      // kernel has to stay in the instruction cache.
#pragma unroll 1
      for (int ph = 0; ph < 5; ++ph) {
        if (ph == 1) {
          commit_wait();
        } else if (ph == 2) {                       // x1 = x + a1 (W2 . t + b2)
          commit_wait();
          float a[32];
          tc::tmem_ld32(lane, a);
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            x1[j] = fmaf(vh[kBlkC + j], a[j] + vh[j], x1[j]);
            v[j] = x1[j];
            if (TRAIN && valid) P.x1[(op - (IO*)P.out) + (size_t)j * HW] = x1[j];
          }
          mix_norm(v, P.eps, mine, other, g);
        } else if (ph >= 3) {                       // GELU of 32 of 64 hidden channels
          const int h0 = 64 * (ph - 3);
          if (ph == 3) commit_wait();
          float a[32];
          tc::tmem_ld32(lane + (uint32_t)h0, a);
#ifdef __CUDA_ARCH__
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            const float2 b = *(const float2*)(vh + 4 * kBlkC + h0 + j);
            const float za = a[j] + b.x, zb = a[j + 1] + b.y;
            const float2 o = gelu_fast2(za, zb);
            if (TRAIN && valid) {
              float* zp = P.z + ((size_t)img * kBlkM + h0) * HW + pos + half_off;
              zp[(size_t)j * HW] = za;
              zp[(size_t)(j + 1) * HW] = zb;
            }
            v[j] = o.x; v[j + 1] = o.y;
          }
#endif
          if (ph == 4) commit_wait();               // the MMAs of the first half have read the operand columns
        }
#ifdef __CUDA_ARCH__
        if (TRAIN && ph < 2) {
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            const float2 o = gelu_fast2(v[j], v[j + 1]);
            v[j] = o.x; v[j + 1] = o.y;
          }
        }
#endif
        mix_stage(lane, v);
        publish();                                  // (the accumulator's first 64 columns have been read by ph = 3)
        if (lead && ok) {
          if (ph == 2) mix_mma<128>(tmem, w3, 0, false);
          else mix_mma<64>(tmem, ph < 2 ? w2 : w4, ph == 1 || ph == 4 ? 64 : 0, ph == 1 || ph == 4);
          tc::mma_commit(done);
        }
        if (ph == 0 || ph == 4) {                   // the second half of t; the next tile
          const IO* q = ph == 0 ? (const IO*)P.t + ((size_t)img * Cin + 64) * HW + pos + half_off : next;
          mix_load<IO>(v, q, HW, ph == 0 ? valid : nvalid);
        }
      }
      commit_wait();
      float a[32];
      tc::tmem_ld32(lane, a);
      if (valid && ok) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          st_io<IO>(op, (size_t)j * HW, fmaf(vh[3 * kBlkC + j], a[j] + vh[2 * kBlkC + j], x1[j]));
      }
    }
    valid = nvalid; img = nimg; pos = npos;
  }
  if (!ok && P.status) atomicExch(P.status, 3);
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(*holder, 512);
}

template <bool POST, typename IO, bool TRAIN = false>
static int launch_mix(const MixParams& P, int sms, cudaStream_t st) {
  const size_t smem = (size_t)(POST ? kPostFloats : kPreFloats) * sizeof(float) + 3 * sizeof(uint64_t) + 8 + 512 * sizeof(float2) + 16;
  const int rc = allow_smem(block_mix_kernel<POST, IO, TRAIN>, smem);
  if (rc != CVB_OK) return rc;
  const long long ntiles = (P.npix + 127) / 128;
  const int grid = (int)(ntiles < sms ? ntiles : sms);     // one block per SM; tiles go round the blocks first
  return launch_chained(block_mix_kernel<POST, IO, TRAIN>, dim3(grid), kMixThreads, smem, st, P);
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
