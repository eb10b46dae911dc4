// Host emulation of the real-plane kernels (csrc/cvb_rp.cuh, cvb_rp_bwd.cuh) -- TEST BUILD ONLY.
// Their bodies are written for one CUDA thread; here every thread of a block is a fiber.  __syncthreads() and the warp
// functions hand over to the next fiber until all threads (all lanes) have arrived, so a barrier or a shuffle that only
// some of them reach is found, as are accesses past either end of a buffer: memory lies between guard zones.
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <ucontext.h>

#include <cmath>
#include <csetjmp>
#include <csignal>
#include <functional>
#include <memory>
#include <stdexcept>
#include <string>
#include <vector>

namespace emu {

struct Index { unsigned x = 0, y = 0, z = 0; };
struct Fiber {
  ucontext_t context;
  std::unique_ptr<char[]> stack;
  Index tid;
  int lane = 0, warp = 0, parity = 0;
  enum { kReady, kBlock, kWarp, kDone } state = kReady;
};
struct WarpSlots { float f[2][32]; int i[2][32]; };

constexpr size_t kStack = 128 * 1024;
Fiber* fiber = nullptr;          // the one running
ucontext_t scheduler;
Index block_index, block_dim, grid_dim;
std::vector<Fiber> fibers;
std::vector<WarpSlots> warps;
const std::function<void()>* body = nullptr;
std::string failure;

void wait(int state) {
  fiber->state = (decltype(fiber->state))state;
  swapcontext(&fiber->context, &scheduler);
}
void sync_block() { wait(Fiber::kBlock); }
// every lane's value, after all lanes have given theirs
template <class T>
T exchange(T (WarpSlots::*slot)[2][32], T v, int from) {
  WarpSlots& w = warps[fiber->warp];
  const int p = fiber->parity;
  fiber->parity ^= 1;            // the other half: a lane that runs ahead must not overwrite what others still read
  (w.*slot)[p][fiber->lane] = v;
  wait(Fiber::kWarp);
  return (w.*slot)[p][from];
}
float shuffle_xor(float v, int mask) { return exchange(&WarpSlots::f, v, fiber->lane ^ mask); }
int any(int pred) {
  WarpSlots& w = warps[fiber->warp];
  const int p = fiber->parity;
  exchange(&WarpSlots::i, pred ? 1 : 0, fiber->lane);
  int r = 0;
  for (int l = 0; l < 32; ++l) r |= w.i[p][l];
  return r;
}
void entry() {
  try {
    (*body)();
  } catch (const std::exception& e) {
    failure = e.what();
  }
  fiber->state = Fiber::kDone;
  swapcontext(&fiber->context, &scheduler);
}

void run_block(int nthr) {
  if ((int)fibers.size() < nthr) fibers.resize(nthr);
  warps.resize(nthr / 32);
  for (int t = 0; t < nthr; ++t) {
    Fiber& f = fibers[t];
    if (!f.stack) f.stack.reset(new char[kStack]);
    f.tid.x = t; f.lane = t & 31; f.warp = t >> 5; f.parity = 0; f.state = Fiber::kReady;
    getcontext(&f.context);
    f.context.uc_stack.ss_sp = f.stack.get();
    f.context.uc_stack.ss_size = kStack;
    f.context.uc_link = nullptr;
    makecontext(&f.context, entry, 0);
  }
  for (;;) {
    int count[4] = {0, 0, 0, 0};
    for (int t = 0; t < nthr; ++t) {
      fiber = &fibers[t];
      if (fiber->state == Fiber::kReady) swapcontext(&scheduler, &fiber->context);
    }
    if (!failure.empty()) {
      const std::string what = failure;
      failure.clear();
      throw std::runtime_error(what);
    }
    for (int t = 0; t < nthr; ++t) ++count[fibers[t].state];
    if (count[Fiber::kDone] == nthr) return;
    bool moved = count[Fiber::kReady] > 0;      // (polling a barrier in shared memory)
    for (int w = 0; w < nthr / 32; ++w) {
      int waiting = 0;
      for (int l = 0; l < 32; ++l) waiting += fibers[32 * w + l].state == Fiber::kWarp;
      if (waiting == 32) {
        for (int l = 0; l < 32; ++l) fibers[32 * w + l].state = Fiber::kReady;
        moved = true;
      }
    }
    if (!moved && count[Fiber::kBlock] == nthr) {
      for (int t = 0; t < nthr; ++t) fibers[t].state = Fiber::kReady;
      moved = true;
    }
    if (!moved) throw std::runtime_error("threads of a block wait for others that never come");
  }
}

// memory between guard zones
class Guarded {
  static constexpr size_t kZone = 4096;
  std::vector<unsigned char> mem;
  size_t n, off;

 public:
  explicit Guarded(size_t bytes) : mem(bytes + 2 * kZone + 256, 0xff), n(bytes) {     // 0xff..: NaN when read
    off = kZone + (256 - ((size_t)mem.data() + kZone) % 256) % 256;
  }
  void* get() { return mem.data() + off; }
  void check(const char* what) const {
    for (size_t i = 0; i < mem.size(); ++i)
      if ((i < off || i >= off + n) && mem[i] != 0xff) throw std::runtime_error(std::string("write past the end of ") + what);
  }
};

template <class F>
void launch(int gx, int gy, int gz, int nthr, F f) {
  const std::function<void()> fn = f;
  body = &fn;
  block_dim = {(unsigned)nthr, 1, 1};
  grid_dim = {(unsigned)gx, (unsigned)gy, (unsigned)gz};
  for (int z = 0; z < gz; ++z)
    for (int y = 0; y < gy; ++y)
      for (int x = 0; x < gx; ++x) {
        block_index = {(unsigned)x, (unsigned)y, (unsigned)z};
        run_block(nthr);
      }
}

}  // namespace emu

#define threadIdx (emu::fiber->tid)
#define blockIdx (emu::block_index)
#define blockDim (emu::block_dim)
#define gridDim (emu::grid_dim)
#define __syncthreads() emu::sync_block()
#define __any_sync(mask, p) emu::any(p)
#define __shfl_xor_sync(mask, v, m) emu::shuffle_xor(v, m)
static inline float __uint_as_float(unsigned v) {
  float f;
  __builtin_memcpy(&f, &v, 4);
  return f;
}
template <class T>
static inline void __stcs(T* p, T v) { *p = v; }
template <class T>
static inline T __ldg(const T* p) { return *p; }

static inline unsigned __float_as_uint(float f) {
  unsigned v;
  __builtin_memcpy(&v, &f, 4);
  return v;
}
static inline int __float2int_rn(float f) { return f != f ? 0 : (int)nearbyintf(f); }
static inline unsigned __byte_perm(unsigned a, unsigned b, unsigned s) {
  const unsigned long long v = ((unsigned long long)b << 32) | a;
  unsigned r = 0;
  for (int i = 0; i < 4; ++i) r |= (unsigned)((v >> (8 * ((s >> (4 * i)) & 7))) & 0xff) << (8 * i);
  return r;
}
static inline unsigned atomicMax(unsigned* p, unsigned v) {
  const unsigned o = *p;
  if (v > o) *p = v;
  return o;
}
static inline int atomicExch(int* p, int v) {
  const int o = *p;
  *p = v;
  return o;
}
static inline unsigned max(unsigned a, unsigned b) { return a > b ? a : b; }
#define __noinline__
#define __syncwarp() emu::wait(emu::Fiber::kWarp)

// Tensor memory, the integer MMA (the second operand in rows of 16 bytes, eight rows a core matrix, K = 32), barriers in
// shared memory and asynchronous copies of cvb_fix.cuh.  MMAs and copies happen at once.  On the GPU MMAs follow each other
// in the order of their issue only where they have the same accumulator and shape; others may overtake one another until a
// commit of theirs has been waited for, so that accumulators which overlap otherwise are an error here.
#include <cstdint>
#include <map>
namespace cvb {
namespace rp {
static int tensor_memory[128][512];
struct Barrier { int pending; long long bytes; uint32_t phase; };
static std::map<uint64_t*, Barrier> barriers;
inline Barrier& barrier(uint64_t* b) {
  auto it = barriers.find(b);
  if (it == barriers.end()) throw std::runtime_error("barrier not initialised");
  return it->second;
}
inline void settle(Barrier& b) {
  if (b.pending < 0) throw std::runtime_error("too many arrivals");
  if (b.pending == 0 && b.bytes == 0) { b.phase ^= 1; b.pending = 1; }
}
inline void fx_init(uint64_t* b) { barriers[b] = {1, 0, 0}; }
inline void fx_init_done() {}
inline void fx_expect(uint64_t* p, uint32_t bytes) { Barrier& b = barrier(p); b.bytes += bytes; --b.pending; settle(b); }
inline void fx_bulk(void* dst, const void* src, uint32_t bytes, uint64_t* p) {
  if (((size_t)dst | (size_t)src | bytes) % 16) throw std::runtime_error("bulk copy alignment");
  memcpy(dst, src, bytes);
  Barrier& b = barrier(p);
  b.bytes -= bytes;
  settle(b);
}
inline bool fx_wait(uint64_t* p, uint32_t parity) {
  for (int i = 0; barrier(p).phase == parity; ++i) {
    if (i > 100000) throw std::runtime_error("a wait that does not end");
    swapcontext(&emu::fiber->context, &emu::scheduler);
  }
  return true;
}
struct Issued { uint32_t d; int n; };
static std::vector<Issued> in_flight;      // since the last commit, which the kernel waits for before it issues again
inline void fx_commit(uint64_t* p) { Barrier& b = barrier(p); --b.pending; settle(b); in_flight.clear(); }
inline unsigned fx_count(unsigned* c) { return (*c)++; }
inline uint32_t fx_elect() { return emu::fiber->lane == 0; }
inline unsigned fx_from_first(unsigned v) { return (unsigned)emu::exchange(&emu::WarpSlots::i, (int)v, 0); }
inline void fx_alloc(uint32_t* holder) {
  if (emu::fiber->lane) return;
  *holder = 0;
  for (auto& l : tensor_memory)
    for (int& v : l) v = 0x5a5a5a5a;
}
inline void fx_free(uint32_t) {}
inline void fx_before_sync() {}
inline void fx_after_sync() {}
struct Operand { const unsigned char* at; int rows; };
inline Operand fx_operand(const unsigned char* b, int brows) { return {b, brows}; }
inline Operand fx_further(Operand b, int bytes) { return {b.at + bytes, b.rows}; }
inline void fx_mma(uint32_t d, uint32_t a, Operand o, int n, bool add, uint32_t elected) {
  if (!elected) return;
  const unsigned char* b = o.at;
  const int brows = o.rows;
  if (n % 16 || n < 16 || n > 256 || d < 256 || d + n > 512 || a + 8 > 256 || (size_t)b % 16) throw std::runtime_error("MMA form");
  for (const Issued& i : in_flight)
    if ((i.d != d || i.n != n) && d < i.d + i.n && i.d < d + n) throw std::runtime_error("MMAs on overlapping accumulators have no order");
  in_flight.push_back({d, n});
  for (int m = 0; m < 128; ++m) {
    const signed char* l = (const signed char*)&tensor_memory[m][a];
    for (int j = 0; j < n; ++j) {
      int sum = add ? tensor_memory[m][d + j] : 0;
      for (int k = 0; k < 32; ++k) sum += (int)l[k] * (int)(signed char)b[(k >> 4) * 16 * brows + j * 16 + (k & 15)];
      tensor_memory[m][d + j] = sum;
    }
  }
}
inline int* tensor_lane(uint32_t t, uint32_t n) {
  if (t >> 16 != (unsigned)(32 * (emu::fiber->warp & 3)) || (t & 0xffff) + n > 512) throw std::runtime_error("tensor-memory access");
  return &tensor_memory[(t >> 16) + emu::fiber->lane][t & 0xffff];
}
template <int N>
inline void fx_ld(uint32_t t, int (&v)[N]) { memcpy(v, tensor_lane(t, N), sizeof(v)); }
inline void fx_ld_wait() {}
template <int N>
inline void fx_st(uint32_t t, const uint32_t (&v)[N]) { memcpy(tensor_lane(t, N), v, sizeof(v)); }
inline void fx_st_wait() {}
template <int BYTES>
inline void fx_copy(void* dst, const void* src, bool ok) {
  if (((size_t)dst | (size_t)src) % BYTES) throw std::runtime_error("asynchronous copy alignment");
  if (ok) memcpy(dst, src, BYTES);
  else memset(dst, 0, BYTES);
}
inline void fx_copies_done() {}
inline float fx_largest(float m, float a, float b) {
  const float v[3] = {m, fabsf(a), fabsf(b)};
  float r = 0.f;
  for (float x : v) r = r != r || x != x ? NAN : x > r ? x : r;
  return r;
}
inline float2 fx_fma2(float2 a, float2 b, float2 c) { return make_float2(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y)); }
inline float2 fx_mul2(float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); }
}  // namespace rp
}  // namespace cvb

#include "../../conversenet_b200/csrc/cvb_rp_plan.h"
#include "../../conversenet_b200/csrc/cvb_rp_bwd.cuh"

using namespace cvb;
using namespace cvb::rp;

namespace {

thread_local std::string message;


void fill_tail(float2* t, const Blob& bl, int h, int w, int r0y, int r1y, int r0x, int r1x) {
  auto unit = [](int m, int N) { return make_float2((float)cos(2.0 * M_PI * m / N), (float)sin(2.0 * M_PI * m / N)); };
  for (int a = 0; a < 2; ++a) {
    const int n = a ? w : h, r0 = a ? r0x : r0y, r1 = a ? r1x : r1y, mp = matrix_width(r0);
    float2 *nat = t + bl.tw + (a ? h : 0), *pos = t + (a ? bl.twx : bl.twy);
    for (int i = 0; i < n; ++i) {
      nat[i] = unit(i, n);
      pos[i] = unit((i / r1) * (i % r1), n);
    }
    float* dm = (float*)(t + (a ? bl.dmx : bl.dmy));
    for (int half = 0; half < 2 && mp; ++half)
      for (int k = 0; k <= r0 / 2; ++k)
        for (int q = 1; q <= mp; ++q) {
          const float2 u = unit((q * k) % r0, r0);
          dm[(half * (r0 / 2 + 1) + k) * mp + q - 1] = q > r0 / 2 ? 0.f : half ? u.y : u.x;
        }
  }
  for (int a = 0; a < 2; ++a) {
    const int n = a ? w : h, nr = fix_rows(n), M = n / 2;
    if (!fix_axis(n, a ? r0x : r0y)) continue;
    unsigned char* out = (unsigned char*)(t + (a ? bl.fixx : bl.fixy));
    for (int par = 0; par < 2; ++par)
      for (int cs = 0; cs < 2; ++cs)
        for (int j = 0; j < nr; ++j)
          for (int q = 0; q < 68; ++q) {
            const int k = 2 * j + par;
            const double u = 2.0 * M_PI * ((q * k) % n) / n;
            double v = k <= M && q <= M / 2 ? (cs ? sin(u) : cos(u)) : 0.0;
            if (q == 0 || 2 * q == M) v *= 0.5;
            if (q >= 64) {
              ((float*)(out + fix_operand(n)))[((par * 2 + cs) * 4 + q - 64) * nr + j] = (float)v;
              continue;
            }
            int m = (int)nearbyint(v / (double)kFixUnit), step;
            const int o = fix_row_offset(nr, par, cs, j, q, step);
            for (int d = 2; d >= 0; --d) {
              const int digit = (signed char)(m & 0xff);
              out[o + d * step] = (unsigned char)digit;
              m = (m - digit) / 256;
            }
          }
  }
}

std::unique_ptr<emu::Guarded> make_table(const float* weight, const float* bias, int C, int k, int s, int h, int w, float eps) {
  int r0y, r1y, r0x, r1x;
  if (!axis_plan(h, r0y, r1y) || !axis_plan(w, r0x, r1x)) return nullptr;
  const Blob bl = blob_layout(C, h, w, r0y, r0x);
  auto mem = std::make_unique<emu::Guarded>(bl.total * sizeof(float2));
  float2* t = (float2*)mem->get();
  TransferParams S;
  memset(&S, 0, sizeof(S));
  S.weight = weight; S.bias = bias; S.C = C; S.k = k; S.s = s; S.h = h; S.w = w; S.eps = eps;
  for (int c = 0; c < C; ++c)
    for (int f = 0; f < w; ++f)
      for (int u = 0; u <= h / 2; ++u) {
        double tr, ti;
        transfer_value_slow(S, c, u, f, tr, ti);
        t[((size_t)c * w + f) * (h / 2 + 1) + u] = make_float2((float)(tr * 0.5 / (h * w)), (float)(ti * 0.5 / (h * w)));
      }
  fill_tail(t, bl, h, w, r0y, r1y, r0x, r1x);
  return mem;
}

void set_vec(Params& P, bool f32) {       // as k_rp.cu
  P.vec = P.p % 2 == 0 && P.W % 2 == 0 && ((size_t)P.x) % (f32 ? 8 : 4) == 0;
  P.vec_out = P.po % 2 == 0 && P.OW % 2 == 0 && ((size_t)P.out) % (f32 ? 8 : 4) == 0;
}

enum Kernel { kColsFwd, kRows, kColsInv };
// (bf16 tensors: one width of the dense stage is enough, the tensor type is met outside it)
template <int MP, typename IO>
void strip_body(const Params& P, Kernel which, float2* sm, int nthr, int grid) {
  constexpr int MAXR = MP ? kMatrixR1 : kAnyRadix;
  if (which == kColsFwd) emu::launch(grid, 1, 1, nthr, [&] { cols_fwd_body<IO, MAXR, MP>(P, sm); });
  if (which == kRows) emu::launch(grid, 1, 1, nthr, [&] { rows_body<MAXR, MP>(P, sm); });
  if (which == kColsInv) emu::launch(grid, 1, 1, nthr, [&] { cols_inv_body<IO, MAXR, MP>(P, sm); });
}
template <typename IO>
void strip(const Params& P, Kernel which, int sms) {
  const Axis& a = which == kRows ? P.ax : P.ay;
  if (takes_fix(P, which, sms)) {
    const size_t bytes = fix_smem(which, a.n);
    emu::Guarded sm(bytes);
    if (bytes > kSmemLimit) throw std::runtime_error("shared memory");
    const int tiles = (fix_lines(which, P) + kFixLines - 1) / kFixLines;
    const int grid = tiles > 2 ? tiles / 2 : tiles;     // blocks walk over several tiles
    auto run = [&](auto extra) {
      constexpr bool E = decltype(extra)::value;
      unsigned char* m = (unsigned char*)sm.get();
      if (which == kColsFwd) emu::launch(grid, 1, 1, kFixThreads, [&] { fix_body<kFixFwd, IO, E>(P, m); });
      if (which == kRows) emu::launch(grid, 1, 1, kFixThreads, [&] { fix_body<kFixRows, IO, E>(P, m); });
      if (which == kColsInv) emu::launch(grid, 1, 1, kFixThreads, [&] { fix_body<kFixInv, IO, E>(P, m); });
    };
    if (a.n >= 256) run(std::true_type());
    else run(std::false_type());
    sm.check("shared memory");
    return;
  }
  const int lines = which == kRows ? P.hh : P.wc, grid = (P.nplane * lines + kLines - 1) / kLines;
  const size_t bytes = which == kRows ? rows_smem(P) : cols_smem(P);
  if (bytes > kSmemLimit) throw std::runtime_error("shared memory");
  emu::Guarded sm(bytes);
  int nthr = strip_threads(P, which == kRows, grid, sms);
  if (a.mp > 44 && nthr > 128) nthr = 128;           // k_rp_matrix.cu
  switch (a.mp) {
    case 0: strip_body<0, IO>(P, which, (float2*)sm.get(), nthr, grid); break;
#define CVB_RP_X(M) case M: if constexpr (sizeof(IO) == 4 || M == 24) strip_body<M, IO>(P, which, (float2*)sm.get(), nthr, grid); break;
      CVB_RP_EACH_WIDTH(CVB_RP_X)
#undef CVB_RP_X
  }
  sm.check("shared memory");
}

template <typename IO>
void forward(Params& P, const Route& r, int sms) {
  const int planes = P.B * P.C;
  set_vec(P, sizeof(IO) == 4);
  if (r.one_block) {
    P.plane0 = 0; P.nplane = planes;
    emu::Guarded sm(plane_smem(P.h, P.w, P.k));
    const bool wide = planes <= sms;
    emu::launch(planes, 1, 1, plane_threads(P, wide ? 512 : 256, planes > 2 * sms),
                [&] { plane_body<IO, kAnyRadix>(P, (float2*)sm.get()); });
    sm.check("shared memory");
    return;
  }
  emu::Guarded ws(r.ws_bytes);
  P.ws = (float2*)ws.get();
  for (int p0 = 0; p0 < planes; p0 += r.chunk) {
    P.plane0 = p0;
    P.nplane = planes - p0 < r.chunk ? planes - p0 : r.chunk;
    if (P.s > 1)
      P.r = P.rsave ? P.rsave + (size_t)p0 * P.h * P.wp : (float*)((char*)ws.get() + (size_t)P.nplane * P.hh * P.wp * sizeof(float2));
    strip<IO>(P, kColsFwd, sms);
    strip<IO>(P, kRows, sms);
    strip<IO>(P, kColsInv, sms);
    if (P.s > 1) {
      emu::Guarded band(kEpiBand);
      emu::launch((P.H + kEpiRows - 1) / kEpiRows, P.nplane, 1, 128, [&] { epilogue_body<IO>(P, (unsigned char*)band.get()); });
      band.check("the epilogue's band");
    }
    ws.check("the workspace");
  }
}

// This file is compiled so that an access at an address its type does not allow (which the GPU refuses) traps.
sigjmp_buf trapped;
void on_trap(int) { siglongjmp(trapped, 1); }
template <class F>
int guarded(F f) {
  struct sigaction act = {}, old;
  act.sa_handler = on_trap;
  sigaction(SIGILL, &act, &old);
  int rc = -1000;
  message.clear();
  try {
    if (sigsetjmp(trapped, 1)) message = "misaligned access";
    else rc = f();
  } catch (const std::exception& e) {
    message = e.what();
  }
  sigaction(SIGILL, &old, nullptr);
  return rc;
}
}  // namespace

extern "C" {

const char* emu_rp_message() { return message.c_str(); }
int emu_rp_plan(int n, int* r0, int* r1) { return axis_plan(n, *r0, *r1) ? matrix_width(*r0) : -1; }
int emu_rp_threads(int planes, int h, int w, int rows, int sms) {
  Params P;
  if (!fill_params(P, nullptr, 1, planes, h, w, 3, 1, 0, 0)) return -1;
  return strip_threads(P, rows, (planes * (rows ? P.hh : P.wc) + kLines - 1) / kLines, sms);
}
int emu_rp_one_block(int B, int C, int H, int W, int s, int p, int sms) {
  return route(B, C, H, W, s, p, sms, false, (size_t)64 << 20).one_block;
}
// both forms fit shared memory at every length they serve
int emu_rp_fits(int h, int w, int planes, int sms) {
  Params P;
  if (!fill_params(P, nullptr, 1, planes, h, w, 3, 1, 0, 0)) return -1;
  const Route r = route(1, planes, h, w, 1, 0, sms, false, (size_t)1 << 40);
  return r.one_block ? plane_smem(h, w, kMaxTaps) <= kSmemLimit : cols_smem(P) <= kSmemLimit && rows_smem(P) <= kSmemLimit;
}

// rsave: r of every plane ([B C][h][wp]) or null; ws_planes: workspace for that many planes (several chunks), 0 = for all
int emu_rp_forward(const void* x, void* out, float* rsave, const float* weight, const float* bias, int B, int C, int H, int W,
                   int k, int s, int p, int mode, float eps, int gelu, int bf16, int force_multi, int ws_planes, int sms) {
  return guarded([&] {
    const int h = H + 2 * p, w = W + 2 * p, e = bf16 ? 2 : 4;
    auto table = make_table(weight, bias, C, k, s, h, w, eps);
    if (!table) return -3;
    const size_t nin = (size_t)B * C * H * W * e, nout = nin * s * s;
    emu::Guarded in(nin), res(nout), keep(rsave ? (size_t)B * C * h * ((w + 1) / 2 * 2) * 4 : 0);
    memcpy(in.get(), x, nin);
    Params P;
    fill_params(P, table->get(), B, C, H, W, k, s, p, mode);
    P.x = in.get(); P.out = res.get(); P.weight = weight; P.gelu = gelu; P.rsave = rsave ? (float*)keep.get() : nullptr;
    const size_t per = ws_plane_bytes(h, w, s);
    const Route r = route(B, C, H, W, s, p, sms, force_multi != 0, ws_planes ? ws_planes * per : (size_t)1 << 40);
    if (bf16) forward<__nv_bfloat16>(P, r, sms);
    else forward<float>(P, r, sms);
    in.check("the input"); res.check("the output"); keep.check("r"); table->check("the table");
    memcpy(out, res.get(), nout);
    if (rsave) memcpy(rsave, keep.get(), (size_t)B * C * h * ((w + 1) / 2 * 2) * 4);
    return 0;
  });
}

// dL/dx, the cross spectrum D ([C][w][hh], summed over its segments, times 4) and, at scale >= 2, the direct tap sums of
// every plane: the kernels of run_bwd without the chain rule
int emu_rp_backward(const float* x, const float* g, const float* r, float* gx, float* D, float* taps, const float* weight,
                    const float* bias, int B, int C, int H, int W, int k, int s, int p, int mode, float eps, int nseg, int sms) {
  return guarded([&] {
    const int h = H + 2 * p, w = W + 2 * p, planes = B * C;
    auto table = make_table(weight, bias, C, k, s, h, w, eps);
    if (!table) return -3;
    Params P;
    fill_params(P, table->get(), B, C, H, W, k, s, p, mode);
    const size_t spec = (size_t)planes * P.hh * P.wp * sizeof(float2);
    emu::Guarded wx(spec), wg(spec), v((size_t)planes * h * w * 4), f((size_t)planes * h * w * 4),
        d((size_t)nseg * C * w * P.hh * sizeof(float2)), tp((size_t)planes * k * k * 4), dx((size_t)planes * H * W * 4);
    Params Y = P;
    Y.s = 1; Y.x = x; Y.ws = (float2*)wx.get(); Y.plane0 = 0; Y.nplane = planes;
    set_vec(Y, true);
    strip<float>(Y, kColsFwd, sms);
    Params Q = P;
    Q.s = 1; Q.ws = (float2*)wg.get(); Q.conj = 1; Q.plane0 = 0; Q.nplane = planes;
    if (s == 1) {
      Q.x = g; Q.pad_mode = 3;
    } else {
      AdjointParams A;
      A.g = g; A.r = r; A.weight = weight; A.v = (float*)v.get(); A.taps = (float*)tp.get();
      A.C = C; A.H = H; A.W = W; A.k = k; A.s = s; A.p = p; A.h = h; A.w = w; A.wp = P.wp;
      auto go = [&](int floats, auto fn) {
        emu::Guarded sm((size_t)floats * 4);
        emu::launch(planes, 1, 1, 256, [&] { fn(A, (float*)sm.get()); });
        sm.check("shared memory");
      };
      switch (s * 16 + k) {
#define X(KK, SS)                                                                                         \
  case SS * 16 + KK:                                                                                      \
    plan_adjoint<KK, SS>(A);                                                                              \
    go(AdjointTile<KK, SS>::floats(A), [](const AdjointParams& a, float* m) { adjoint_epilogue_body<KK, SS>(a, m); }); \
    break;
        X(2, 2) X(3, 2) X(5, 2) X(7, 3) X(3, 4)
#undef X
        default: go(8, [](const AdjointParams& a, float* m) { adjoint_epilogue_any(a, m); });
      }
      v.check("v"); tp.check("taps");
      Q.x = A.v; Q.H = h; Q.W = w; Q.p = 0; Q.pad_mode = 0;
      memcpy(taps, tp.get(), (size_t)planes * k * k * 4);
    }
    set_vec(Q, true);
    strip<float>(Q, kColsFwd, sms);
    if (!D) {          // dL/dx alone
      strip<float>(Q, kRows, sms);
    } else {
      BwdParams R;
      R.P = Q; R.wx = (const float2*)wx.get(); R.D = (float2*)d.get(); R.nseg = nseg; R.solve = 1;
      const size_t tile = ((size_t)P.pitch * kLines + 1) & ~(size_t)1;
      emu::Guarded sm(3 * tile * sizeof(float2) + (P.ax.mp ? matrix_entries(P.ax.r0) : 0) * sizeof(float));
      const int rows = (P.hh + kLines - 1) / kLines;
      switch (P.ax.mp) {
        case 0: emu::launch(rows, C, nseg, 128, [&] { rows_bwd_body<kAnyRadix, 0>(R, (float2*)sm.get()); }); break;
#define CVB_RP_X(M) case M: emu::launch(rows, C, nseg, 128, [&] { rows_bwd_body<kMatrixR1, M>(R, (float2*)sm.get()); }); break;
          CVB_RP_EACH_WIDTH(CVB_RP_X)
#undef CVB_RP_X
      }
      sm.check("shared memory"); d.check("D"); wg.check("the workspace");
      const float2* dd = (const float2*)d.get();
      const size_t n = (size_t)C * w * P.hh;
      for (size_t i = 0; i < n; ++i) {
        double a = 0, b = 0;
        for (int sg = 0; sg < nseg; ++sg) { a += dd[sg * n + i].x; b += dd[sg * n + i].y; }
        D[2 * i] = (float)a; D[2 * i + 1] = (float)b;
      }
    }
    const bool direct = s == 1 && p == 0;
    Params O = Q;
    O.po = 0; O.OH = h; O.OW = w; O.out = direct ? dx.get() : f.get();
    set_vec(O, true);
    strip<float>(O, kColsInv, sms);
    if (!direct) {
      PadAdjointParams A;
      A.f = (const float*)f.get(); A.g = s > 1 ? g : nullptr; A.gx = (float*)dx.get();
      A.H = H; A.W = W; A.s = s; A.p = p; A.h = h; A.w = w; A.pad_mode = mode;
      emu::launch((H * W + 1023) / 1024, planes, 1, 256, [&] { pad_adjoint_body(A); });
    }
    dx.check("dL/dx"); f.check("the solved cotangent"); wx.check("the workspace");
    memcpy(gx, dx.get(), (size_t)planes * H * W * 4);
    return 0;
  });
}
}
