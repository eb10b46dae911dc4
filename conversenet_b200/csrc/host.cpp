// Host side of the Python entry points: argument checks, allocation, stream look-up and the C ABI calls of one layer or
// one block in a single native call.  A small layer runs in a few microseconds on the GPU; going through Python and
// ctypes for every buffer and argument took 22 us a call, four times the kernel (24 x 20 planes, 64 channels).
//
// The C ABI is reached through the function addresses of the library that the package loaded (init()), so there is one
// copy of it in the process.  Only tensors' public C++ interface is used.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <ATen/ATen.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdlib>
#include <cstring>
#include <memory>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/converse_b200.h"

namespace {

struct Api {
  decltype(&cvb_strerror) strerror_ = nullptr;
  decltype(&cvb_last_cuda_error) last_cuda_error = nullptr;
  decltype(&cvb_transfer_bytes) transfer_bytes = nullptr;
  decltype(&cvb_build_transfer) build_transfer = nullptr;
  decltype(&cvb_build_x0_table) build_x0_table = nullptr;
  decltype(&cvb_converse2d_workspace_bytes) workspace_bytes = nullptr;
  decltype(&cvb_converse2d_fwd) converse2d_fwd = nullptr;
  decltype(&cvb_block_pack_bytes) block_pack_bytes = nullptr;
  decltype(&cvb_block_pack) block_pack = nullptr;
  decltype(&cvb_block_pre_fwd) block_pre = nullptr;
  decltype(&cvb_block_post_fwd) block_post = nullptr;
  decltype(&cvb_converse2d_train_workspace_bytes) train_workspace_bytes = nullptr;
  decltype(&cvb_converse2d_fwd_train) fwd_train = nullptr;
  decltype(&cvb_converse2d_bwd_workspace_bytes) bwd_workspace_bytes = nullptr;
  decltype(&cvb_converse2d_bwd) bwd = nullptr;
  decltype(&cvb_block_pre_train) block_pre_train = nullptr;
  decltype(&cvb_block_post_train) block_post_train = nullptr;
  decltype(&cvb_block_grad_floats) block_grad_floats = nullptr;
  decltype(&cvb_block_bwd_workspace_bytes) block_bwd_workspace = nullptr;
  decltype(&cvb_block_bwd) block_bwd = nullptr;
  decltype(&cvb_takes_pairs) takes_pairs = nullptr;
  decltype(&cvb_plane_transfer_bytes) plane_bytes = nullptr;
  decltype(&cvb_build_plane_transfer) build_plane = nullptr;
  decltype(&cvb_pair_transfer_bytes) pair_bytes = nullptr;
  decltype(&cvb_build_pair_transfer) build_pair = nullptr;
  decltype(&cvb_pair_workspace_bytes) pair_workspace_bytes = nullptr;
  decltype(&cvb_pair_fwd) pair_fwd = nullptr;
  decltype(&cvb_takes_planes) takes_planes = nullptr;
  decltype(&cvb_plane_workspace_bytes) plane_workspace_bytes = nullptr;
  decltype(&cvb_plane_fwd) plane_fwd = nullptr;
} api;

struct Failed : std::runtime_error { using std::runtime_error::runtime_error; };

void check(int rc, const char* what) {
  if (rc == 0) return;
  std::string m = std::string(what) + " failed: " + api.strerror_(rc);
  if (rc == CVB_ERR_CUDA) m += " (cudaError " + std::to_string(api.last_cuda_error()) + ")";
  throw Failed(m);
}

const at::Tensor& tensor(PyObject* o, const char* what) {
  if (!THPVariable_Check(o)) throw Failed(std::string(what) + " must be a tensor");
  return THPVariable_Unpack(o);
}
const at::Tensor& cuda_tensor(PyObject* o, const char* what) {
  const at::Tensor& t = tensor(o, what);
  if (!t.is_cuda()) throw Failed("Converse2D needs a CUDA tensor; this build has no CPU path");
  return t;
}
long integer(PyObject* o) {
  const long v = PyLong_AsLong(o);
  if (v == -1 && PyErr_Occurred()) throw std::invalid_argument("");
  return v;
}
double real(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw std::invalid_argument("");
  return v;
}
int io_type(const at::Tensor& t) {
  if (t.scalar_type() == at::kFloat) return CVB_F32;
  if (t.scalar_type() == at::kBFloat16) return CVB_BF16;
  throw Failed("Converse2D supports float32 and bfloat16 tensors, got torch." + std::string(
      t.scalar_type() == at::kHalf ? "float16" : t.scalar_type() == at::kDouble ? "float64" : toString(t.scalar_type())));
}
int pad_mode(PyObject* o) {
  const char* s = PyUnicode_Check(o) ? PyUnicode_AsUTF8(o) : nullptr;
  if (s) {
    if (!std::strcmp(s, "circular")) return CVB_PAD_CIRCULAR;
    if (!std::strcmp(s, "replicate")) return CVB_PAD_REPLICATE;
    if (!std::strcmp(s, "reflect")) return CVB_PAD_REFLECT;
    if (!std::strcmp(s, "constant")) return CVB_PAD_CONSTANT;
  }
  throw Failed("unknown padding_mode '" + std::string(s ? s : "?") + "'");
}
void* stream(const at::Tensor& t) { return (void*)c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
at::Tensor bytes_like(const at::Tensor& t, size_t n) {
  return at::empty({(int64_t)n}, t.options().dtype(at::kByte).requires_grad(false));
}
// a parameter as contiguous fp32 (itself when it already is)
at::Tensor f32(const at::Tensor& t) {
  if (t.scalar_type() == at::kFloat && t.is_contiguous()) return t;
  return t.detach().to(at::kFloat).contiguous();
}

// What `table` is and who reads it: the table of build_transfer for any batch (or one that serves this batch as well); the pair
// table alone, for the pair kernels; the real-plane one (or one that begins with it), for the real planes where
// cvb_takes_planes prefers them
enum Form { kAnyBatch = 0, kPairTable = 1, kPlaneTable = 2 };
at::Tensor forward(const at::Tensor& x, const at::Tensor& table, const at::Tensor& wf, int k, int s, int p, int mode,
                   int gelu, at::Tensor out, int form) {
  const int B = (int)x.size(0), C = (int)x.size(1), H = (int)x.size(2), W = (int)x.size(3), io = io_type(x);
  if (!out.defined()) out = at::empty({B, C, (int64_t)H * s, (int64_t)W * s}, x.options().requires_grad(false));
  const size_t full = sizeof(float) * 2 * (size_t)C * (H + 2 * p) * (W + 2 * p);   // below that: no pair table in it
  const bool pairs = form == kPairTable, planes = !pairs && api.takes_planes(B, C, H + 2 * p, W + 2 * p, s);
  if ((size_t)table.numel() < full && !(planes && form == kPlaneTable) &&
      (pairs || api.takes_pairs(B, H + 2 * p, W + 2 * p, s) == 2))
    throw Failed("the transfer table was built for another batch size");
  const size_t ws = pairs    ? api.pair_workspace_bytes(B, C, H, W, s, p)
                    : planes ? api.plane_workspace_bytes(B, C, H, W, s, p)
                             : api.workspace_bytes(B, C, H, W, s, p, io);
  at::Tensor w;
  if (ws) w = bytes_like(x, ws);
  check((pairs ? api.pair_fwd : planes ? api.plane_fwd : api.converse2d_fwd)(x.data_ptr(), out.data_ptr(), table.data_ptr(), (const float*)wf.data_ptr(), B, C,
                                                    H, W, k, s, p, mode, io, gelu, ws ? w.data_ptr() : nullptr, ws, stream(x)),
        "cvb_converse2d_fwd");
  return out;
}

// The calling thread without the interpreter's lock: allocations and launches may wait (a full launch queue, an allocator
// that has to synchronise), and other Python threads go on meanwhile.  Arguments are read before, results wrapped after.
struct Unlocked {
  PyThreadState* state = PyEval_SaveThread();
  ~Unlocked() { PyEval_RestoreThread(state); }
};

template <class F>
PyObject* guarded(F f) {
  try {
    return f();
  } catch (const Failed& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  } catch (const c10::Error& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
  } catch (const std::exception& e) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}
void want(Py_ssize_t n, Py_ssize_t m) {
  if (n != m) throw Failed("wrong number of arguments");
}

// converse2d(x, table, weight_f32, kernel_size, scale, padding, padding_mode, fuse_gelu, out or None, form)
PyObject* py_converse2d(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    want(n, 10);
    const at::Tensor& x0 = cuda_tensor(a[0], "x");
    if (x0.dim() != 4) throw Failed("x must be (B,C,H,W)");
    const c10::cuda::CUDAGuard dev(x0.device());
    const at::Tensor &table = tensor(a[1], "table"), &wf = tensor(a[2], "weight");
    const int k = (int)integer(a[3]), s = (int)integer(a[4]), p = (int)integer(a[5]), mode = pad_mode(a[6]), form = (int)integer(a[9]);
    const int gelu = PyObject_IsTrue(a[7]);
    at::Tensor out;
    if (a[8] != Py_None) out = tensor(a[8], "out");
    {
      const Unlocked unlocked;
      out = forward(x0.is_contiguous() ? x0 : x0.contiguous(), table, wf, k, s, p, mode, gelu, std::move(out), form);
    }
    return THPVariable_Wrap(std::move(out));
  });
}

// takes_pairs(B, h, w, scale) -> cvb_takes_pairs; with the channels behind them, 0 where cvb_takes_planes answers 1
PyObject* py_takes_pairs(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n != 5) want(n, 4);
    const int B = (int)integer(a[0]), h = (int)integer(a[1]), w = (int)integer(a[2]), s = (int)integer(a[3]);
    const int pairs = api.takes_pairs(B, h, w, s);
    return PyLong_FromLong(pairs == 2 && n == 5 && api.takes_planes(B, (int)integer(a[4]), h, w, s) ? 0 : pairs);
  });
}

// build_transfer(weight, bias, scale, eps, h, w, x0_term, which) -> (table, weight as contiguous fp32 (C,k,k))
// which: 0 tables for every batch, 1 the pair table, 2 the real-plane table (where there is one; else the pair table)
PyObject* py_build_transfer(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    want(n, 8);
    const at::Tensor &w = tensor(a[0], "weight"), &b = tensor(a[1], "bias");
    const long s = integer(a[2]), h = integer(a[4]), wd = integer(a[5]);
    if (!w.is_cuda()) throw Failed("Converse2D parameters must live on a CUDA device");
    if (w.dim() != 4 || w.size(0) != 1) throw Failed("weight must be (1,C,kh,kw)");
    const int C = (int)w.size(1), k = (int)w.size(2);
    if (w.size(3) != k) throw Failed("only square kernels are supported");
    if (b.dim() != 4 || b.size(0) != 1 || b.size(1) != C || b.size(2) != 1 || b.size(3) != 1)
      throw Failed("bias must be (1,C,1,1)");
    if (s < 1) throw Failed("scale must be >= 1");
    const bool x0 = PyObject_IsTrue(a[6]);
    const long which = integer(a[7]);
    const size_t plane = api.plane_bytes(C, (int)h, (int)wd);
    size_t bytes = which == 1 ? api.pair_bytes(C, (int)h, (int)wd) : api.transfer_bytes(C, (int)h, (int)wd);
    auto fn = which == 1 ? api.build_pair : x0 ? api.build_x0_table : api.build_transfer;
    // every batch: the real-plane table alone serves the sizes whose blob is no larger than the pair table
    if (plane && !x0 && which != 1 && (which == 2 || bytes <= api.pair_bytes(C, (int)h, (int)wd))) {
      bytes = plane;
      fn = api.build_plane;
    }
    if (!bytes) throw Failed("padded plane " + std::to_string(h) + "x" + std::to_string(wd) + " is not supported by the FFT engine");
    const c10::cuda::CUDAGuard dev(w.device());
    const float eps = (float)real(a[3]);
    at::Tensor table, wf;
    {
      const Unlocked unlocked;
      wf = f32(w.detach()).view({C, k, k});
      const at::Tensor bf = f32(b.detach());
      table = bytes_like(w, bytes);
      check(fn((const float*)wf.data_ptr(), (const float*)bf.data_ptr(), C, k, (int)s, (int)h, (int)wd, eps,
               table.data_ptr(), stream(w)),
            "cvb_build_transfer");
    }
    return Py_BuildValue("(NN)", THPVariable_Wrap(table), THPVariable_Wrap(wf));
  });
}

// backend() -> CONVERSE2D_BACKEND of the environment, None when it is not set.  os.environ writes through to it; its own
// look-up takes 0.7 us of a small call's 10.
PyObject* py_backend(PyObject*, PyObject* const*, Py_ssize_t) {
  const char* v = std::getenv("CONVERSE2D_BACKEND");
  if (!v || !*v) Py_RETURN_NONE;
  return PyUnicode_DecodeFSDefault(v);
}

// state(t, ...) -> bytes: storage addresses and version counters, equal bytes = unmodified tensors (None allowed), then
// (eight bytes) the current stream of the first CUDA tensor's device.  None
// when a tensor was made in inference mode: it counts no versions, so a change in place could not be seen and nothing
// derived from it may be kept.
PyObject* py_state(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    for (Py_ssize_t i = 0; i < n; ++i)
      if (a[i] != Py_None && THPVariable_Check(a[i]) && THPVariable_Unpack(a[i]).is_inference()) Py_RETURN_NONE;
    PyObject* o = PyBytes_FromStringAndSize(nullptr, n * 16 + 8);
    if (!o) return nullptr;
    char* d = PyBytes_AS_STRING(o);
    void* st = nullptr;
    bool found = false;
    for (Py_ssize_t i = 0; i < n; ++i) {
      int64_t v[2] = {0, 0};
      if (a[i] != Py_None && THPVariable_Check(a[i])) {
        const at::Tensor& t = THPVariable_Unpack(a[i]);
        v[0] = (int64_t)t.data_ptr();
        v[1] = (int64_t)t._version();
        if (!found && t.is_cuda()) st = stream(t), found = true;
      }
      std::memcpy(d + 16 * i, v, 16);
    }
    std::memcpy(d + 16 * n, &st, 8);
    return o;
  });
}

void cuda(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return;
  (void)cudaGetLastError();
  throw Failed(std::string(what) + " failed: " + cudaGetErrorString(e));
}
bool capturing(cudaStream_t st) {
  cudaStreamCaptureStatus s = cudaStreamCaptureStatusNone;
  cuda(cudaStreamIsCapturing(st, &s), "cudaStreamIsCapturing");
  return s != cudaStreamCaptureStatusNone;
}

// Events that no Ready holds any more, at most kSpareEvents a device; the interpreter's lock guards them.  (Training lays its
// tables out at every step: making and destroying an event each time takes 1 us.)
constexpr size_t kSpareEvents = 32;
std::vector<cudaEvent_t>& spare_events(int device) {
  static std::vector<cudaEvent_t> spare[64];
  return spare[device & 63];
}
// What a kept value needs beside itself: an event behind the work that makes it, and the storages whose addresses name it
struct Ready {
  int device;
  cudaEvent_t event = nullptr;
  std::vector<c10::Storage> pins;
  explicit Ready(int d) : device(d) {
    auto& spare = spare_events(device);
    if (spare.empty()) {
      cuda(cudaEventCreateWithFlags(&event, cudaEventDisableTiming), "cudaEventCreate");
    } else {
      event = spare.back();
      spare.pop_back();
    }
  }
  ~Ready() {
    auto& spare = spare_events(device);
    if (spare.size() < kSpareEvents) spare.push_back(event);
    else cudaEventDestroy(event);
  }
};

// ready(t, param, ...) -> a Ready behind the work on the current stream of t's device so far, holding the parameters'
// storages; None during a capture
PyObject* py_ready(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n < 1) throw Failed("wrong number of arguments");
    const at::Tensor& t = cuda_tensor(a[0], "tensor");
    const c10::cuda::CUDAGuard dev(t.device());
    const cudaStream_t st = (cudaStream_t)stream(t);
    if (capturing(st)) Py_RETURN_NONE;
    auto r = std::make_unique<Ready>((int)t.device().index());
    for (Py_ssize_t i = 1; i < n; ++i)
      if (a[i] != Py_None) r->pins.push_back(tensor(a[i], "parameter").storage());
    cuda(cudaEventRecord(r->event, st), "cudaEventRecord");
    PyObject* o = PyCapsule_New(r.get(), "cvb.ready", [](PyObject* c) { delete (Ready*)PyCapsule_GetPointer(c, "cvb.ready"); });
    if (o) r.release();
    return o;
  });
}

// join(ready, t, ...): the current stream waits for its event, and the allocator learns that it uses the tensors.  False,
// and nothing done, during a capture.
PyObject* py_join(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n < 2) throw Failed("wrong number of arguments");
    const Ready* r = (const Ready*)PyCapsule_GetPointer(a[0], "cvb.ready");
    if (!r) throw std::invalid_argument("ready");
    const at::Tensor& t = cuda_tensor(a[1], "tensor");
    const c10::cuda::CUDAGuard dev(t.device());
    const c10::cuda::CUDAStream st = c10::cuda::getCurrentCUDAStream(t.device().index());
    if (capturing(st.stream())) Py_RETURN_FALSE;
    cuda(cudaStreamWaitEvent(st.stream(), r->event, 0), "cudaStreamWaitEvent");
    for (Py_ssize_t i = 1; i < n; ++i)
      c10::cuda::CUDACachingAllocator::recordStream(cuda_tensor(a[i], "tensor").storage().data_ptr(), st);
    Py_RETURN_TRUE;
  });
}

// block_pack(ln1.weight, ln1.bias, w1, b1, w2, b2, alpha1, ln2.weight, ln2.bias, w3, b3, w4, b4, alpha2) -> packed weights
PyObject* py_block_pack(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    want(n, 14);
    at::Tensor t[14], pack;
    const float* q[14];
    for (int i = 0; i < 14; ++i)
      if (a[i] != Py_None) t[i] = cuda_tensor(a[i], "parameter");
    const c10::cuda::CUDAGuard dev(t[2].device());
    {
      const Unlocked unlocked;
      for (int i = 0; i < 14; ++i) {
        if (t[i].defined()) t[i] = f32(t[i]);
        q[i] = t[i].defined() ? (const float*)t[i].data_ptr() : nullptr;
      }
      pack = bytes_like(t[2], api.block_pack_bytes());
      check(api.block_pack(q[0], q[1], q[2], q[3], q[4], q[5], q[6], q[7], q[8], q[9], q[10], q[11], q[12], q[13],
                           pack.data_ptr(), stream(pack)),
            "cvb_block_pack");
    }
    return THPVariable_Wrap(std::move(pack));
  });
}

// block(x, table, weight_f32, pack, kernel_size, padding, padding_mode, eps1, eps2, form) -> ConverseBlock.forward(x)
PyObject* py_block(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    want(n, 10);
    const at::Tensor& x0 = cuda_tensor(a[0], "x");
    if (x0.dim() != 4) throw Failed("x must be (B,C,H,W)");
    const c10::cuda::CUDAGuard dev(x0.device());
    const at::Tensor &table = tensor(a[1], "table"), &wf = tensor(a[2], "weight"), &pack = tensor(a[3], "pack");
    const int B = (int)x0.size(0), C = (int)x0.size(1), H = (int)x0.size(2), W = (int)x0.size(3), io = io_type(x0);
    const int k = (int)integer(a[4]), p = (int)integer(a[5]), mode = pad_mode(a[6]);
    const float eps1 = (float)real(a[7]), eps2 = (float)real(a[8]);
    const int form = (int)integer(a[9]);
    at::Tensor out;
    {
      const Unlocked unlocked;
      const at::Tensor x = x0.is_contiguous() ? x0 : x0.contiguous();
      const auto opt = x.options().requires_grad(false);
      void* st = stream(x);
      at::Tensor t = at::empty({B, 2 * C, H, W}, opt);
      check(api.block_pre(x.data_ptr(), t.data_ptr(), pack.data_ptr(), eps1, B, H * W, io, st), "cvb_block_pre_fwd");
      t = forward(t, table, wf, k, 1, p, mode, 1, at::Tensor(), form);
      out = at::empty({B, C, H, W}, opt);
      check(api.block_post(t.data_ptr(), x.data_ptr(), out.data_ptr(), pack.data_ptr(), eps2, B, H * W, io, st),
            "cvb_block_post_fwd");
    }
    return THPVariable_Wrap(std::move(out));
  });
}

// train_forward(x, table, weight_f32, kernel_size, scale, padding, padding_mode) -> (out, r or None); None when the
// gradient kernels give no parameter gradients for the shape (nothing would read r)
PyObject* py_train_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    want(n, 7);
    const at::Tensor& x0 = cuda_tensor(a[0], "x");
    if (x0.dim() != 4) throw Failed("x must be (B,C,H,W)");
    const c10::cuda::CUDAGuard dev(x0.device());
    const at::Tensor &table = tensor(a[1], "table"), &wf = tensor(a[2], "weight");
    const int B = (int)x0.size(0), C = (int)x0.size(1), H = (int)x0.size(2), W = (int)x0.size(3), io = io_type(x0);
    const int k = (int)integer(a[3]), s = (int)integer(a[4]), p = (int)integer(a[5]), mode = pad_mode(a[6]);
    if (!api.bwd_workspace_bytes(B, C, H, W, k, s, p, 0, 1)) Py_RETURN_NONE;
    at::Tensor out, r;
    int rc = CVB_OK;
    if (s == 1) {        // nothing to keep
      const Unlocked unlocked;
      out = forward(x0.is_contiguous() ? x0 : x0.contiguous(), table, wf, k, s, p, mode, 0, at::Tensor(), kPlaneTable);
    } else {
      const Unlocked unlocked;
      const at::Tensor x = x0.is_contiguous() ? x0 : x0.contiguous();
      at::Tensor w;
      out = at::empty({B, C, (int64_t)H * s, (int64_t)W * s}, x.options().requires_grad(false));
      r = at::empty({B, C, H + 2 * p, (W + 2 * p + 1) / 2 * 2}, x.options().dtype(at::kFloat).requires_grad(false));
      const size_t ws = api.train_workspace_bytes(B, C, H, W, s, p);
      if (ws) w = bytes_like(x, ws);
      rc = api.fwd_train(x.data_ptr(), out.data_ptr(), table.data_ptr(), (const float*)wf.data_ptr(),
                         (float*)r.data_ptr(), B, C, H, W, k, s, p, mode, io, ws ? w.data_ptr() : nullptr, ws, stream(x));
      if (rc != CVB_ERR_UNSUPPORTED_SIZE) check(rc, "cvb_converse2d_fwd_train");
    }
    if (rc == CVB_ERR_UNSUPPORTED_SIZE) Py_RETURN_NONE;
    PyObject* rr = Py_None;
    if (s > 1) rr = THPVariable_Wrap(r);
    else Py_INCREF(rr);
    return Py_BuildValue("(NN)", THPVariable_Wrap(out), rr);
  });
}

// backward(x or None, g, r or None, table, weight, bias, (B,C,H,W) of x, scale, padding, padding_mode, eps, want_x,
// want_params) -> (gx, gw, gb), unwanted ones None; None when the kernels do not take the shape
PyObject* py_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    want(n, 13);
    const at::Tensor &g0 = cuda_tensor(a[1], "g"), &w0 = tensor(a[4], "weight"), &b0 = tensor(a[5], "bias");
    const c10::cuda::CUDAGuard dev(g0.device());
    int d[4];
    for (int i = 0; i < 4; ++i) d[i] = (int)integer(PyTuple_GetItem(a[6], i));
    const int B = d[0], C = d[1], H = d[2], W = d[3], k = (int)w0.size(-1);
    const int s = (int)integer(a[7]), p = (int)integer(a[8]), mode = pad_mode(a[9]);
    const float eps = (float)real(a[10]);
    const bool wx = PyObject_IsTrue(a[11]), wp = PyObject_IsTrue(a[12]);
    const size_t ws = api.bwd_workspace_bytes(B, C, H, W, k, s, p, wx, wp);
    if (!ws) Py_RETURN_NONE;
    const at::Tensor& table = tensor(a[3], "table");
    at::Tensor x, r, gx, gw, gb;
    if (wp) x = cuda_tensor(a[0], "x").detach();
    if (a[2] != Py_None) r = tensor(a[2], "r");
    {
      const Unlocked unlocked;
      const at::Tensor g = f32(g0.detach()), wf = f32(w0.detach()), bf = f32(b0.detach());
      if (wp) x = f32(x);
      const auto opt = g.options().requires_grad(false);
      if (wx) gx = at::empty({B, C, H, W}, opt);
      if (wp) {
        gw = at::empty(w0.sizes(), opt);
        gb = at::empty(b0.sizes(), opt);
      }
      at::Tensor work = bytes_like(g, ws);
      auto ptr = [](const at::Tensor& t) { return t.defined() ? (float*)t.data_ptr() : nullptr; };
      check(api.bwd(ptr(x), ptr(g), ptr(r), table.data_ptr(), ptr(wf), ptr(bf), ptr(gx), ptr(gw), ptr(gb), B, C, H, W, k, s, p,
                    mode, eps, work.data_ptr(), ws, stream(g)),
            "cvb_converse2d_bwd");
    }
    auto wrap = [](const at::Tensor& t) -> PyObject* {
      if (t.defined()) return THPVariable_Wrap(t);
      Py_RETURN_NONE;
    };
    return Py_BuildValue("(NNN)", wrap(gx), wrap(gw), wrap(gb));
  });
}

// block_train(x, table, weight_f32, pack, kernel_size, padding, padding_mode, eps1, eps2) -> (out, t1, z1, u, x1, z3), the
// last five for block_backward; None when the gradient kernels do not take the shape
PyObject* py_block_train(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    want(n, 9);
    const at::Tensor& x0 = cuda_tensor(a[0], "x");
    const c10::cuda::CUDAGuard dev(x0.device());
    const at::Tensor &table = tensor(a[1], "table"), &wf = tensor(a[2], "weight"), &pack = tensor(a[3], "pack");
    const int B = (int)x0.size(0), C = (int)x0.size(1), H = (int)x0.size(2), W = (int)x0.size(3);
    const int k = (int)integer(a[4]), p = (int)integer(a[5]), mode = pad_mode(a[6]);
    const float eps1 = (float)real(a[7]), eps2 = (float)real(a[8]);
    if (!api.block_bwd_workspace(B, H, W, k, p)) Py_RETURN_NONE;
    at::Tensor t1, z1, u, x1, z3, out;
    {
      const Unlocked unlocked;
      const at::Tensor x = f32(x0.detach());
      const auto opt = x.options().requires_grad(false);
      void* st = stream(x);
      t1 = at::empty({B, 2 * C, H, W}, opt), z1 = at::empty({B, 2 * C, H, W}, opt), u = at::empty({B, 2 * C, H, W}, opt);
      x1 = at::empty({B, C, H, W}, opt), z3 = at::empty({B, 2 * C, H, W}, opt), out = at::empty({B, C, H, W}, opt);
      check(api.block_pre_train((const float*)x.data_ptr(), (float*)t1.data_ptr(), (float*)z1.data_ptr(), pack.data_ptr(), eps1,
                                B, H * W, st), "cvb_block_pre_train");
      forward(t1, table, wf, k, 1, p, mode, 0, u, kPlaneTable);
      check(api.block_post_train((const float*)u.data_ptr(), (const float*)x.data_ptr(), (float*)out.data_ptr(),
                                 (float*)x1.data_ptr(), (float*)z3.data_ptr(), pack.data_ptr(), eps2, B, H * W, st),
            "cvb_block_post_train");
    }
    return Py_BuildValue("(NNNNNN)", THPVariable_Wrap(out), THPVariable_Wrap(t1), THPVariable_Wrap(z1), THPVariable_Wrap(u),
                         THPVariable_Wrap(x1), THPVariable_Wrap(z3));
  });
}

// block_backward(x, t1, z1, u, x1, z3, g, table, conv_weight, conv_bias, params (14 tensors or None), eps1, eps2, conv_eps,
// padding, padding_mode) -> [gx, gconv_w, gconv_b, the 14 parameter gradients (None for an absent alpha)]
PyObject* py_block_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    want(n, 16);
    at::Tensor in[7], par[14];
    const float* pp[14];
    for (int i = 0; i < 7; ++i) in[i] = cuda_tensor(a[i], "tensor").detach();
    const c10::cuda::CUDAGuard dev(in[0].device());
    for (int i = 0; i < 14; ++i) {
      PyObject* o = PyTuple_GetItem(a[10], i);
      if (!o) throw std::invalid_argument("params");
      if (o != Py_None) par[i] = tensor(o, "parameter").detach();
    }
    const at::Tensor &table = tensor(a[7], "table"), &cw = tensor(a[8], "weight"), &cb = tensor(a[9], "bias");
    cvb_block_bwd_args A;
    std::memset(&A, 0, sizeof(A));
    A.eps1 = (float)real(a[11]); A.eps2 = (float)real(a[12]); A.conv_eps = (float)real(a[13]);
    A.k = (int)cw.size(-1); A.p = (int)integer(a[14]); A.pad_mode = pad_mode(a[15]);
    at::Tensor gx, gcw, gcb, gp;
    {
      const Unlocked unlocked;
      const float* ip[7];
      for (int i = 0; i < 7; ++i) {
        in[i] = f32(in[i]);
        ip[i] = (const float*)in[i].data_ptr();
      }
      for (int i = 0; i < 14; ++i) {
        if (par[i].defined()) par[i] = f32(par[i]);
        pp[i] = par[i].defined() ? (const float*)par[i].data_ptr() : nullptr;
      }
      const at::Tensor cwf = f32(cw.detach()), cbf = f32(cb.detach());
      const auto opt = in[0].options().requires_grad(false);
      A.x = ip[0]; A.t1 = ip[1]; A.z1 = ip[2]; A.u = ip[3]; A.x1 = ip[4]; A.z3 = ip[5]; A.g = ip[6];
      A.table = table.data_ptr();
      A.conv_w = (const float*)cwf.data_ptr(); A.conv_b = (const float*)cbf.data_ptr();
      A.ln1_w = pp[0]; A.ln1_b = pp[1]; A.w1 = pp[2]; A.b1 = pp[3]; A.w2 = pp[4]; A.b2 = pp[5]; A.alpha1 = pp[6];
      A.ln2_w = pp[7]; A.ln2_b = pp[8]; A.w3 = pp[9]; A.b3 = pp[10]; A.w4 = pp[11]; A.b4 = pp[12]; A.alpha2 = pp[13];
      A.B = (int)in[0].size(0); A.H = (int)in[0].size(2); A.W = (int)in[0].size(3);
      gx = at::empty(in[0].sizes(), opt), gcw = at::empty(cw.sizes(), opt), gcb = at::empty(cb.sizes(), opt);
      gp = at::empty({(int64_t)api.block_grad_floats()}, opt);
      const size_t ws = api.block_bwd_workspace(A.B, A.H, A.W, A.k, A.p);
      at::Tensor work = bytes_like(in[0], ws ? ws : 1);
      A.gx = (float*)gx.data_ptr(); A.gconv_w = (float*)gcw.data_ptr(); A.gconv_b = (float*)gcb.data_ptr();
      A.gparams = (float*)gp.data_ptr();
      A.workspace = work.data_ptr(); A.workspace_bytes = ws; A.stream = stream(in[0]);
      check(api.block_bwd(&A), "cvb_block_bwd");
    }
    PyObject* out = PyList_New(17);
    PyList_SET_ITEM(out, 0, THPVariable_Wrap(gx));
    PyList_SET_ITEM(out, 1, THPVariable_Wrap(gcw));
    PyList_SET_ITEM(out, 2, THPVariable_Wrap(gcb));
    static const int64_t size[7] = {64, 64, 8192, 128, 8192, 64, 64};
    int64_t off = 0;
    for (int i = 0; i < 14; ++i) {
      PyObject* o = Py_None;
      if (pp[i]) o = THPVariable_Wrap(gp.narrow(0, off, size[i % 7]).view(par[i].sizes()));
      else Py_INCREF(o);
      PyList_SET_ITEM(out, 3 + i, o);
      off += size[i % 7];
    }
    return out;
  });
}

// init(address of each C ABI function in the order of `names`)
PyObject* py_init(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    want(n, 30);
    void* p[30];
    for (int i = 0; i < 30; ++i) p[i] = PyLong_AsVoidPtr(a[i]);
    int i = 0;
    auto set = [&](auto& f) { f = (std::decay_t<decltype(f)>)p[i++]; };
    set(api.strerror_); set(api.last_cuda_error); set(api.transfer_bytes); set(api.build_transfer); set(api.build_x0_table);
    set(api.workspace_bytes); set(api.converse2d_fwd); set(api.block_pack_bytes); set(api.block_pack); set(api.block_pre);
    set(api.block_post); set(api.train_workspace_bytes); set(api.fwd_train); set(api.bwd_workspace_bytes); set(api.bwd);
    set(api.block_pre_train); set(api.block_post_train); set(api.block_grad_floats); set(api.block_bwd_workspace);
    set(api.block_bwd); set(api.takes_pairs); set(api.plane_bytes); set(api.build_plane); set(api.pair_bytes);
    set(api.build_pair); set(api.pair_workspace_bytes); set(api.pair_fwd);
    set(api.takes_planes); set(api.plane_workspace_bytes); set(api.plane_fwd);
    Py_RETURN_NONE;
  });
}

PyMethodDef methods[] = {
    {"init", (PyCFunction)(void (*)(void))py_init, METH_FASTCALL, nullptr},
    {"converse2d", (PyCFunction)(void (*)(void))py_converse2d, METH_FASTCALL, nullptr},
    {"takes_pairs", (PyCFunction)(void (*)(void))py_takes_pairs, METH_FASTCALL, nullptr},
    {"build_transfer", (PyCFunction)(void (*)(void))py_build_transfer, METH_FASTCALL, nullptr},
    {"state", (PyCFunction)(void (*)(void))py_state, METH_FASTCALL, nullptr},
    {"backend", (PyCFunction)(void (*)(void))py_backend, METH_FASTCALL, nullptr},
    {"ready", (PyCFunction)(void (*)(void))py_ready, METH_FASTCALL, nullptr},
    {"join", (PyCFunction)(void (*)(void))py_join, METH_FASTCALL, nullptr},
    {"block_pack", (PyCFunction)(void (*)(void))py_block_pack, METH_FASTCALL, nullptr},
    {"train_forward", (PyCFunction)(void (*)(void))py_train_forward, METH_FASTCALL, nullptr},
    {"backward", (PyCFunction)(void (*)(void))py_backward, METH_FASTCALL, nullptr},
    {"block_train", (PyCFunction)(void (*)(void))py_block_train, METH_FASTCALL, nullptr},
    {"block_backward", (PyCFunction)(void (*)(void))py_block_backward, METH_FASTCALL, nullptr},
    {"block", (PyCFunction)(void (*)(void))py_block, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
  PyObject* m = PyModule_Create(&module);
  if (!m) return nullptr;
  PyObject* names = Py_BuildValue("(ssssssssssssssssssssssssssssss)", "cvb_strerror", "cvb_last_cuda_error", "cvb_transfer_bytes",
                                  "cvb_build_transfer", "cvb_build_x0_table", "cvb_converse2d_workspace_bytes",
                                  "cvb_converse2d_fwd", "cvb_block_pack_bytes", "cvb_block_pack", "cvb_block_pre_fwd",
                                  "cvb_block_post_fwd", "cvb_converse2d_train_workspace_bytes",
                                  "cvb_converse2d_fwd_train", "cvb_converse2d_bwd_workspace_bytes", "cvb_converse2d_bwd",
                                  "cvb_block_pre_train", "cvb_block_post_train", "cvb_block_grad_floats",
                                  "cvb_block_bwd_workspace_bytes", "cvb_block_bwd", "cvb_takes_pairs",
                                  "cvb_plane_transfer_bytes", "cvb_build_plane_transfer", "cvb_pair_transfer_bytes",
                                  "cvb_build_pair_transfer", "cvb_pair_workspace_bytes", "cvb_pair_fwd",
                                  "cvb_takes_planes", "cvb_plane_workspace_bytes", "cvb_plane_fwd");
  if (!names || PyModule_AddObject(m, "names", names) < 0) return nullptr;
  return m;
}
