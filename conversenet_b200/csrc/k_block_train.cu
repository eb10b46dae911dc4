// Gradients of ConverseBlock's channel mixing (models/util_converse.py:278-293 under autograd), fp32.  With xh, rstd the
// normalised values of a LayerNorm, z1, z3 the hidden layers before their GELUs and u the Converse2D output:
//   g_z3 = (a2 W4)^T g . gelu'(z3)                    block_grad_kernel<UP>     64 -> 128 channels
//   g_x1 = g + LN2'((W3 gamma2)^T g_z3)               block_grad_kernel<DOWN>  128 ->  64
//   g_u  = (a1 W2)^T g_x1 . gelu'(u)                  UP, then the gradient of Converse2D (k_rp_bwd.cu) gives g_t
//   g_z1 = g_t . gelu'(z1);  g_x = g_x1 + LN1'((W1 gamma1)^T g_z1)               DOWN
// and every parameter gradient follows from four contractions over the pixels (wgrad_kernel), each 64 x 128 with the sums
// of both operands:  g (x) gelu(z3),  xh2 (x) g_z3,  g_x1 (x) gelu(u),  xh1 (x) g_z1.
// The contractions over channels run as in k_block_mlp.cu (two groups of 256 threads, operand in tensor memory) with TF32
// hi + lo; those over pixels too, their sums in fp32 registers.
#include "../../include/converse_b200.h"
#include "cvb_internal.h"
#include "cvb_mix.cuh"

namespace cvb {

// ---- weights of the four channel contractions, split and in operand layout: 2 kW floats each, in the order of their use
struct GradPackParams {
  const float *ln1_w, *w1, *w2, *a1, *ln2_w, *w3, *w4, *a2;
  float* out;
};
__global__ void __launch_bounds__(256) block_grad_pack_kernel(const GradPackParams P) {
  const int which = blockIdx.x >> 4, slice = blockIdx.x & 15;
  float* hi = P.out + which * 2 * kW;
  for (int i = slice * (kW / 16) + threadIdx.x; i < (slice + 1) * (kW / 16); i += 256) {
    float v, a, b;
    int idx;
    if ((which & 1) == 0) {         // UP: rows n = hidden channel, K = 64 channels c
      const int n = i >> 6, c = i & 63;
      const float* w = which == 0 ? P.w4 : P.w2;
      const float* al = which == 0 ? P.a2 : P.a1;
      v = w[c * kBlkM + n] * (al ? al[c] : 1.0f);
      idx = pack_index(kBlkM, n, c);
    } else {                        // DOWN: rows n = channel, K = 128 hidden channels
      const int n = i >> 7, j = i & 127;
      v = (which == 1 ? P.w3 : P.w1)[j * kBlkC + n] * (which == 1 ? P.ln2_w : P.ln1_w)[n];
      idx = pack_index(kBlkC, n, j);
    }
    tc::split_tf32(v, a, b);
    hi[idx] = a;
    hi[kW + idx] = b;
  }
}

// gelu'(v) = Phi(v) + v phi(v), Phi by the erfc polynomial of gelu_fast2
__device__ __forceinline__ float gelu_grad(float v) {
  const float u = fminf(fabsf(v), 6.2225397f);
  float q = -2.3622640075e-06f;
  q = fmaf(q, u, 3.3874740336e-05f);
  q = fmaf(q, u, -1.6080242733e-04f);
  q = fmaf(q, u, -1.9633368643e-04f);
  q = fmaf(q, u, 7.1384621134e-03f);
  q = fmaf(q, u, -5.2546291581e-02f);
  q = fmaf(q, u, -4.5919230672e-01f);
  q = fmaf(q, u, -1.1511069657e+00f);
  const float h = exp2f(fmaf(q, u, -1.0f));                                  // erfc / 2
  const float phi = 0.3989422804f * exp2f(-0.7213475204f * v * v);
  return fmaf(v, phi, v >= 0.f ? 1.0f - h : h);
}

struct BlockGradParams {
  const float* in;      // UP (B,64,HW); DOWN (B,128,HW)
  const float* z;       // UP: gelu' of it multiplies the result.  DOWN: of it multiplies the input, or null
  float* gz;            // DOWN with z: the multiplied input, kept
  const float* x;       // DOWN: input of the LayerNorm
  const float* res;     // DOWN: added to the result
  float* xh;            // DOWN: normalised x, kept
  float* out;
  const float* pack;
  float eps;
  int HW;
  long long npix;
  int* status;
};

template <bool DOWN>
__global__ void __launch_bounds__(kMixThreads, 1) block_grad_kernel(const __grid_constant__ BlockGradParams P) {
  extern __shared__ __align__(128) float msm[];
  float* wts = msm;
  uint64_t* bars = (uint64_t*)(msm + 2 * kW);       // MMA of group 0, 1; weights
  uint32_t* holder = (uint32_t*)(bars + 3);
  float2* halves = (float2*)(holder + 2);           // [group][half][pixel], twice
  const int tid = threadIdx.x, warp = tid >> 5, g = tid >> 8, m = tid & 127, hf = (tid >> 7) & 1;
  const bool lead = (tid & 255) == 0;
  float2* mine = halves + (g * 2 + hf) * 128 + m;
  const float2* other = halves + (g * 2 + (hf ^ 1)) * 128 + m;
  if (tid == 0) {
    for (int i = 0; i < 3; ++i) mbar_init(&bars[i], 1);
    mbar_fence_init();
    mbar_expect_tx(&bars[2], 2 * kW * 4);
    bulk_g2s(wts, P.pack, 2 * kW * 4, &bars[2]);
  }
  if (warp == 0) tc::tmem_alloc(holder, 512);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *holder + 256u * (uint32_t)g;
  const uint32_t lane = tmem + ((uint32_t)((warp & 3) * 32) << 16) + 32u * (uint32_t)hf;
  uint64_t* done = &bars[g];
  uint32_t uses = 0;
  bool ok = mbar_wait_bounded(&bars[2], 0, kWaitLimit);
  auto commit_wait = [&]() {
    if (ok) ok = mbar_wait_bounded(done, uses & 1u, kWaitLimit);
    uses += 1;
    tc::fence_after_sync();
  };
  auto publish = [&]() {
    tc::fence_before_sync();
    mix_bar(g);
    tc::fence_after_sync();
  };
  const long long ntiles = (P.npix + 127) / 128;
  const int HW = P.HW;
  for (long long tile = blockIdx.x + (long long)g * gridDim.x; tile < ntiles; tile += 2ll * gridDim.x) {
    const long long pix = tile * 128 + m;
    const bool valid = pix < P.npix;
    const long long img = valid ? pix / HW : 0;
    const int pos = valid ? (int)(pix - img * HW) : 0;
    const size_t at64 = ((size_t)img * kBlkC + 32 * hf) * HW + pos, at128 = ((size_t)img * kBlkM + 32 * hf) * HW + pos;
    float v[32];
    if constexpr (!DOWN) {
      mix_load<float>(v, P.in + at64, HW, valid);
      mix_stage(lane, v);
      publish();
      if (lead && ok) { mix_mma<128>(tmem, wts, 0, false, 1u); tc::mma_commit(done); }
      const size_t at = ((size_t)img * kBlkM + 64 * hf) * HW + pos;
      mix_load<float>(v, P.z + at, HW, valid);
      commit_wait();
#pragma unroll 1
      for (int c0 = 0; c0 < 64; c0 += 32) {
        float a[32];
        tc::tmem_ld32(lane + (uint32_t)(32 * hf + c0), a);
#pragma unroll
        for (int j = 0; j < 32; ++j) a[j] *= gelu_grad(v[j]);
        if (c0 == 0) mix_load<float>(v, P.z + at + (size_t)32 * HW, HW, valid);
        if (valid && ok) {
#pragma unroll
          for (int j = 0; j < 32; ++j) P.out[at + (size_t)(c0 + j) * HW] = a[j];
        }
      }
    } else {
#pragma unroll 1
      for (int ph = 0; ph < 2; ++ph) {
        const size_t at = at128 + (size_t)(64 * ph) * HW;
        mix_load<float>(v, P.in + at, HW, valid);
        if (P.z) {
          float z[32];
          mix_load<float>(z, P.z + at, HW, valid);
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            v[j] *= gelu_grad(z[j]);
            if (valid) P.gz[at + (size_t)j * HW] = v[j];
          }
        }
        if (ph) commit_wait();
        mix_stage(lane, v);
        publish();
        if (lead && ok) { mix_mma<64>(tmem, wts, 64 * ph, ph != 0, 1u); tc::mma_commit(done); }
      }
      mix_load<float>(v, P.x + at64, HW, valid);
      const float rstd = mix_norm(v, P.eps, mine, other, g);
      commit_wait();
      float a[32];
      tc::tmem_ld32(lane, a);
      float s0 = 0.f, s1 = 0.f, q0 = 0.f, q1 = 0.f;
#pragma unroll
      for (int j = 0; j < 32; j += 2) {
        s0 += a[j]; s1 += a[j + 1];
        q0 = fmaf(a[j], v[j], q0); q1 = fmaf(a[j + 1], v[j + 1], q1);
      }
      mine[512] = make_float2(s0 + s1, q0 + q1);
      mix_bar(g);
      const float2 o = other[512];
      const float mg = (s0 + s1 + o.x) * (1.0f / 64), mq = (q0 + q1 + o.y) * (1.0f / 64);
      if (valid && ok) {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          P.xh[at64 + (size_t)j * HW] = v[j];
          P.out[at64 + (size_t)j * HW] = fmaf(rstd, a[j] - fmaf(v[j], mq, mg), P.res[at64 + (size_t)j * HW]);
        }
      }
    }
  }
  if (!ok && P.status) atomicExch(P.status, 3);
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(*holder, 512);
}

template <bool DOWN>
static int launch_grad(const BlockGradParams& P, int sms, cudaStream_t st) {
  const size_t smem = 2 * kW * sizeof(float) + 3 * sizeof(uint64_t) + 8 + 1024 * sizeof(float2) + 16;
  CVB_CUDA(cudaFuncSetAttribute(block_grad_kernel<DOWN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const long long ntiles = (P.npix + 127) / 128;
  const int grid = (int)(ntiles < sms ? ntiles : sms);
  block_grad_kernel<DOWN><<<grid, kMixThreads, smem, st>>>(P);
  CVB_CUDA(cudaGetLastError());
  return CVB_OK;
}

// ------------------------------------------------------------------ contractions over the pixels
// out[p][q] = sum over pixels of P[p] Q[q], 64 x 128, and the sums of every P[p] and Q[q]; Q optionally through GELU.
// A block takes 32-pixel tiles blockIdx.x, + gridDim.x, ...: its threads split the 192 channels' values into TF32 hi + lo
// (exact to 2^-22 of a value) in shared memory, channels as rows and pixels along K, and one tile's MMAs (Q in the 128 rows
// of tensor memory; hi hi in 64 columns, hi lo + lo hi in another 64) run while the next is split.  The accumulators are read
// and added to fp32 sums in registers after every tile: the tensor cores cut what they add off instead of rounding it, which over
// four additions (eight of the small products) stays below what rounding the sum of a block's thousand pixels costs: gradients of w1 to w4 of a block of
// 8 x 64 x 64 are within 5.7e-7 to 8.5e-7 of fp64 (8.0e-7 to 1.1e-6 with fp32 products on the CUDA cores).  32768 pixels,
// the four contractions: 50 us, 99 on the CUDA cores (which waited for the port to shared memory); 100 MB take 15 us.  The
// erf of the GELUs, the split and its stores are the larger part of a tile.  An infinity among the operands makes the sums that it meets
// NaN (hi - hi), not infinite.
constexpr int kGOut = kBlkC * kBlkM + kBlkC + kBlkM;
constexpr int kGThreads = 512, kGRows = 128, kGGroup = kGRows * 16 + 16;   // bytes of four pixels of 128 rows (+ 16: banks)
constexpr int kGOperand = 8 * kGGroup, kGBuffer = 3 * kGOperand;           // Q hi, Q lo, [P hi | P lo]
struct WgradParams {
  const float* p[4];
  const float* q[4];
  int gelu[4];
  float* part;          // [4][blocks][kGOut]
  int HW;
  long long npix;
  int* status;
};
__global__ void __launch_bounds__(kGThreads, 2) wgrad_kernel(const __grid_constant__ WgradParams W) {
  extern __shared__ __align__(128) char gsm[];
  uint64_t* done = (uint64_t*)(gsm + 2 * kGBuffer);
  uint32_t* holder = (uint32_t*)(done + 1);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, which = blockIdx.y;
  const int HW = W.HW;
  const bool gelu = W.gelu[which] != 0;
  if (tid == 0) {
    mbar_init(done, 1);
    mbar_fence_init();
  }
  if (warp == 0) tc::tmem_alloc(holder, 128);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *holder;
  // this thread's part of the result: row q = 32 (warp & 3) + lane, sixteen columns p
  const int p0 = 16 * (warp >> 2);
  const uint32_t mine = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)p0;
  float acc[16], sum[12], r[12];
#pragma unroll
  for (int i = 0; i < 16; ++i) acc[i] = 0.f;
#pragma unroll
  for (int i = 0; i < 12; ++i) sum[i] = 0.f;
  const long long ntiles = (W.npix + 31) / 32;
  // channels warp, warp + 16, ... of P and then of Q at pixel `lane` of tile t
  auto load = [&](long long t) {
    const long long pix = t * 32 + lane;
    const bool in = t < ntiles && pix < W.npix;
    const long long img = !in ? 0 : W.npix <= 0x7fffffff ? (unsigned)pix / (unsigned)HW : pix / HW;
    const int pos = in ? (int)(pix - img * HW) : 0;
    const float* a = W.p[which] + ((size_t)img * kBlkC + warp) * HW + pos;
    const float* b = W.q[which] + ((size_t)img * kBlkM + warp) * HW + pos;
    const size_t step = (size_t)16 * HW;
#pragma unroll
    for (int i = 0; i < 4; ++i) r[i] = in ? a[i * step] : 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) r[4 + i] = in ? b[i * step] : 0.f;
  };
  bool ok = true;
  uint32_t uses = 0;
  auto drain = [&]() {
    if (ok) ok = mbar_wait_bounded(done, uses & 1u, kWaitLimit);
    uses += 1;
    tc::fence_after_sync();
#pragma unroll
    for (int c = 0; c < 16; c += 8) {
      uint32_t x[8], y[8];
      tc::tmem_ld8(mine + (uint32_t)c, x);
      tc::tmem_ld8(mine + 64u + (uint32_t)c, y);
      tc::tmem_wait_ld();
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[c + j] += __uint_as_float(x[j]) + __uint_as_float(y[j]);
    }
    tc::fence_before_sync();
  };
  load(blockIdx.x);
  int it = 0;
  for (long long t = blockIdx.x; t < ntiles; t += gridDim.x, ++it) {
    char* buf = gsm + (it & 1) * kGBuffer + (lane >> 2) * kGGroup + (lane & 3) * 4 + warp * 16;
#pragma unroll
    for (int i = 0; i < 12; ++i) {
      const float v = i >= 4 && gelu ? gelu_erf(r[i]) : r[i];
      sum[i] += v;
      float hi, lo;
      tc::split_tf32(v, hi, lo);
      char* dst = buf + (i < 4 ? 2 * kGOperand + i * 256 : (i - 4) * 256);      // 16 rows further
      *(float*)dst = hi;
      *(float*)(dst + (i < 4 ? 64 * 16 : kGOperand)) = lo;
    }
    load(t + gridDim.x);
    tc::fence_proxy_async();
    if (it > 0) drain();                       // the other buffer is free then, and so are the accumulators
    __syncthreads();
    if (warp == 0) {
      tc::fence_after_sync();
      const uint32_t e = tc::elect_one() & tc::from_first(ok ? 1u : 0u);
      const char* base = gsm + (it & 1) * kGBuffer;
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        const uint64_t qh = tc::smem_desc(base + 2 * ks * kGGroup, kGGroup, 128);
        const uint64_t ql = tc::smem_desc(base + kGOperand + 2 * ks * kGGroup, kGGroup, 128);
        const uint64_t ph = tc::smem_desc(base + 2 * kGOperand + 2 * ks * kGGroup, kGGroup, 128);
        const uint64_t pl = tc::smem_desc(base + 2 * kGOperand + 2 * ks * kGGroup + 64 * 16, kGGroup, 128);
        // (all of one shape: MMAs of another one on the same columns would have no order among them)
        constexpr uint32_t idesc = tc::idesc_tf32(128, 64, false, false);
        tc::mma_tf32_elected(tmem, qh, ph, idesc, ks > 0 ? 1u : 0u, e);
        tc::mma_tf32_elected(tmem + 64u, qh, pl, idesc, ks > 0 ? 1u : 0u, e);
        tc::mma_tf32_elected(tmem + 64u, ql, ph, idesc, 1u, e);
      }
      if (e) tc::mma_commit(done);
    }
  }
  if (it > 0) drain();
  if (!ok && W.status) atomicExch(W.status, 3);
  float* o = W.part + ((size_t)which * gridDim.x + blockIdx.x) * kGOut;
  const int q = 32 * (warp & 3) + lane;
#pragma unroll
  for (int j = 0; j < 16; ++j) o[(p0 + j) * kBlkM + q] = acc[j];
#pragma unroll
  for (int i = 0; i < 12; ++i) {
    float x = sum[i];
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) x += __shfl_xor_sync(0xffffffffu, x, k);
    if (lane == 0) o[kBlkC * kBlkM + warp + 16 * i] = x;
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, 128);
}
// sums of the blocks' parts -> part of block 0
__global__ void __launch_bounds__(128) wgrad_sum_kernel(float* part, int blocks) {
  const int i = blockIdx.x * 128 + threadIdx.x;
  if (i >= kGOut) return;
  float* p = part + (size_t)blockIdx.y * blocks * kGOut + i;
  float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
  int b = 0;
  for (; b + 3 < blocks; b += 4) {
    s0 += p[(size_t)b * kGOut]; s1 += p[(size_t)(b + 1) * kGOut];
    s2 += p[(size_t)(b + 2) * kGOut]; s3 += p[(size_t)(b + 3) * kGOut];
  }
  for (; b < blocks; ++b) s0 += p[(size_t)b * kGOut];
  *p = (s0 + s1) + (s2 + s3);
}
struct FinishBlockParams {
  const float* part;
  int blocks;
  const float *ln1_w, *ln1_b, *w1, *w2, *b2, *a1, *ln2_w, *ln2_b, *w3, *w4, *b4, *a2;
  float* out;           // gradients one after the other: ln1_w ln1_b w1 b1 w2 b2 a1 ln2_w ln2_b w3 b3 w4 b4 a2
};
// grid (4 contractions, 8 slices)
__global__ void __launch_bounds__(256) finish_block_kernel(const FinishBlockParams F) {
  const int which = blockIdx.x, slice = blockIdx.y, tid = threadIdx.x;
  const float* R = F.part + (size_t)which * F.blocks * kGOut;     // [64][128]
  const float *SP = R + kBlkC * kBlkM, *SQ = SP + kBlkC;
  constexpr int half = 2 * kBlkC + kW + kBlkM + kW + kBlkC + kBlkC;   // ln w b1 | w2 b2 a1
  const bool second = which < 2;                                       // contractions 0, 1 belong to conv2
  float* o = F.out + (second ? half : 0);
  float *dlw = o, *dlb = o + kBlkC, *dwu = o + 2 * kBlkC, *dbu = dwu + kW;       // LN, up-convolution
  // order of a half: conv1: ln1 w1 b1 w2 b2 a1; conv2: ln2 w3 b3 w4 b4 a2
  float *dwd = dbu + kBlkM, *dbd = dwd + kW, *da = dbd + kBlkC;
  if ((which & 1) == 0) {
    const float* w = which == 0 ? F.w4 : F.w2;
    const float* b = which == 0 ? F.b4 : F.b2;
    const float* al = which == 0 ? F.a2 : F.a1;
    for (int i = slice * (kW / 8) + tid; i < (slice + 1) * (kW / 8); i += 256) dwd[i] = R[i] * (al ? al[i >> 7] : 1.0f);
    const int c = slice * 8 + (tid >> 5), ln = tid & 31;
    float s = 0.f;
    for (int j = ln; j < kBlkM; j += 32) s = fmaf(w[c * kBlkM + j], R[c * kBlkM + j], s);
    for (int x = 16; x > 0; x >>= 1) s += __shfl_xor_sync(0xffffffffu, s, x);
    if (ln == 0) {
      da[c] = fmaf(b[c], SP[c], s);
      dbd[c] = SP[c] * (al ? al[c] : 1.0f);
    }
  } else {
    const float* w = which == 1 ? F.w3 : F.w1;
    const float* ga = which == 1 ? F.ln2_w : F.ln1_w;
    const float* be = which == 1 ? F.ln2_b : F.ln1_b;
    for (int i = slice * (kW / 8) + tid; i < (slice + 1) * (kW / 8); i += 256) {
      const int n = i >> 6, k = i & 63;
      dwu[i] = fmaf(ga[k], R[k * kBlkM + n], be[k] * SQ[n]);
    }
    if (slice == 0)
      for (int n = tid; n < kBlkM; n += 256) dbu[n] = SQ[n];
    const int k = slice * 8 + (tid >> 5), ln = tid & 31;
    float s = 0.f, t = 0.f;
    for (int n = ln; n < kBlkM; n += 32) {
      s = fmaf(w[n * kBlkC + k], R[k * kBlkM + n], s);
      t = fmaf(w[n * kBlkC + k], SQ[n], t);
    }
    for (int x = 16; x > 0; x >>= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, x);
      t += __shfl_xor_sync(0xffffffffu, t, x);
    }
    if (ln == 0) { dlw[k] = s; dlb[k] = t; }
  }
}

// ------------------------------------------------------------------ one backward call
static int wgrad_blocks(long long npix, int sms) {
  const long long t = (npix + 31) / 32;
  const int most = sms / 2 > 1 ? sms / 2 : 1;       // four contractions x sms / 2 blocks = two blocks on every SM
  return (int)(t < most ? t : most);
}
size_t block_grad_floats() { return 2 * (2 * (size_t)kBlkC + 2 * kW + kBlkM + 2 * kBlkC); }

struct BlockGradPlan { size_t pack, gz3, gx1, gu, gz1, xh1, xh2, part, conv, total; };
static BlockGradPlan plan_block_grad(int B, int HW, size_t conv_ws, int sms) {
  auto up = [](size_t n) { return (n + 255) / 256 * 256; };
  const size_t n = (size_t)B * HW * sizeof(float);
  BlockGradPlan b;
  size_t at = 0;
  auto take = [&](size_t bytes) { const size_t o = at; at += up(bytes); return o; };
  b.pack = take(8 * (size_t)kW * sizeof(float));
  b.gz3 = take(kBlkM * n);
  b.gx1 = take(kBlkC * n);
  b.gu = take(kBlkM * n);
  b.gz1 = take(kBlkM * n);
  b.xh1 = take(kBlkC * n);
  b.xh2 = take(kBlkC * n);
  b.part = take((size_t)4 * wgrad_blocks((long long)B * HW, sms) * kGOut * sizeof(float));
  b.conv = take(conv_ws);
  b.total = at;
  return b;
}
size_t block_grad_workspace(int B, int HW, size_t conv_ws, int sms) { return plan_block_grad(B, HW, conv_ws, sms).total; }

int run_block_grad(const cvb_block_bwd_args& A, size_t conv_ws, int sms, int* status, cudaStream_t st,
                   int (*conv)(const cvb_block_bwd_args&, const float* gu, float* gt, void* ws, size_t bytes)) {
  const int HW = A.H * A.W;
  const long long npix = (long long)A.B * HW;
  const BlockGradPlan b = plan_block_grad(A.B, HW, conv_ws, sms);
  if (!A.workspace || A.workspace_bytes < b.total) return CVB_ERR_WORKSPACE;
  char* base = (char*)A.workspace;
  auto at = [&](size_t o) { return (float*)(base + o); };
  const GradPackParams K = {A.ln1_w, A.w1, A.w2, A.alpha1, A.ln2_w, A.w3, A.w4, A.alpha2, at(b.pack)};
  block_grad_pack_kernel<<<64, 256, 0, st>>>(K);
  CVB_CUDA(cudaGetLastError());
  BlockGradParams P;
  P.HW = HW; P.npix = npix; P.status = status;
  P.gz = nullptr; P.xh = nullptr; P.x = nullptr; P.res = nullptr; P.eps = 0.f;
  int rc;
  P.in = A.g; P.z = A.z3; P.out = at(b.gz3); P.pack = at(b.pack);
  if ((rc = launch_grad<false>(P, sms, st)) != CVB_OK) return rc;
  P.in = at(b.gz3); P.z = nullptr; P.x = A.x1; P.res = A.g; P.xh = at(b.xh2); P.out = at(b.gx1); P.eps = A.eps2;
  P.pack = at(b.pack) + 2 * kW;
  if ((rc = launch_grad<true>(P, sms, st)) != CVB_OK) return rc;
  P.in = at(b.gx1); P.z = A.u; P.out = at(b.gu); P.pack = at(b.pack) + 4 * kW;
  if ((rc = launch_grad<false>(P, sms, st)) != CVB_OK) return rc;
  float* gt = at(b.gz1);                            // becomes g_z1 in place
  if ((rc = conv(A, at(b.gu), gt, base + b.conv, conv_ws)) != CVB_OK) return rc;
  P.in = gt; P.z = A.z1; P.gz = gt; P.x = A.x; P.res = at(b.gx1); P.xh = at(b.xh1); P.out = A.gx; P.eps = A.eps1;
  P.pack = at(b.pack) + 6 * kW;
  if ((rc = launch_grad<true>(P, sms, st)) != CVB_OK) return rc;
  WgradParams W;
  const float* ps[4] = {A.g, at(b.xh2), at(b.gx1), at(b.xh1)};
  const float* qs[4] = {A.z3, at(b.gz3), A.u, gt};
  for (int i = 0; i < 4; ++i) { W.p[i] = ps[i]; W.q[i] = qs[i]; W.gelu[i] = i == 0 || i == 2; }
  W.part = at(b.part); W.HW = HW; W.npix = npix; W.status = status;
  const int blocks = wgrad_blocks(npix, sms);
  constexpr int smem = 2 * kGBuffer + 16;
  CVB_CUDA(cudaFuncSetAttribute(wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  wgrad_kernel<<<dim3(blocks, 4), kGThreads, smem, st>>>(W);
  CVB_CUDA(cudaGetLastError());
  wgrad_sum_kernel<<<dim3((kGOut + 127) / 128, 4), 128, 0, st>>>(W.part, blocks);
  CVB_CUDA(cudaGetLastError());
  const FinishBlockParams F = {W.part, blocks, A.ln1_w, A.ln1_b, A.w1, A.w2, A.b2, A.alpha1, A.ln2_w, A.ln2_b, A.w3,
                               A.w4, A.b4, A.alpha2, A.gparams};
  finish_block_kernel<<<dim3(4, 8), 256, 0, st>>>(F);
  CVB_CUDA(cudaGetLastError());
  return CVB_OK;
}

}  // namespace cvb
