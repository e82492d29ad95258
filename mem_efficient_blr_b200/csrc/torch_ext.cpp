// Thin PyTorch C++ extension over the C ABI of libblr_b200.so: the operators as TORCH_LIBRARY ops (CUDA + Meta
// kernels), so that an eager call costs a dispatcher hop instead of a ctypes conversion per argument, and a compiled
// graph calls straight into C++.  No arithmetic lives here: tensors in, pointers and sizes to the C entry points,
// tensors out.  Beside the dispatcher's operators the file is a Python module of the same calls without the dispatcher (see
// "direct calls" below).  The signatures are those of the Python layer's operators (ops.py), which mirror the reference's
// operator functions one level up (triton_funcs/*.py entry points; models/wrappers.py:143-146 resolves them by name).
//
// Scratch: one workspace per (device, stream), from cudaMalloc through the library (PyTorch's CUDA-graph memory pools
// are no home for a long-lived buffer); while a stream capture is under way the buffer comes from the capture's pool.
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/Exceptions.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/record_function.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <torch/library.h>

#include <map>
#include <mutex>
#include <utility>
#include <vector>

#include "blr_b200.h"

namespace {

struct Scratch {
  void* ptr = nullptr;
  size_t bytes = 0;
  at::Tensor holder;  // set when the buffer had to come from torch's allocator (stream capture under way)
  // A workspace whose head has been zeroed by captured work only, of which nobody knows whether it ever runs: every further capture
  // (`capture`: the last one) records the zeroing again, until a call outside of captures has done it.
  bool unset = false;
  unsigned long long capture = 0;
};

std::mutex g_mu;
std::map<std::pair<int, cudaStream_t>, Scratch> g_ws, g_staging;
std::vector<Scratch> g_retired;

void check_rc(int rc) { TORCH_CHECK(rc == 0, "blr_b200 error ", rc, ": ", blr_last_error()); }

// The capture under way on a stream; 0: none.
unsigned long long capture_of(cudaStream_t st) {
  cudaStreamCaptureStatus s = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  return cudaStreamGetCaptureInfo(st, &s, &id) == cudaSuccess && s != cudaStreamCaptureStatusNone ? id : 0;
}

struct Room {
  void* ptr;
  size_t bytes;
};

// The buffer of (device, stream), at least `need` bytes.  By value, read under the lock: another thread may grow the entry right after.
// Grows geometrically.
Room scratch(std::map<std::pair<int, cudaStream_t>, Scratch>& reg, int dev, cudaStream_t st, size_t need, bool is_ws) {
  std::lock_guard<std::mutex> lock(g_mu);
  Scratch& s = reg[{dev, st}];
  if (s.bytes >= need && !s.unset) return {s.ptr, s.bytes};
  const unsigned long long capture = capture_of(st);
  if (s.bytes < need) {
    size_t cap = need < (size_t(1) << 20) ? (size_t(1) << 20) : need;
    if (cap < 2 * s.bytes) cap = 2 * s.bytes;
    if (s.ptr != nullptr) {
      // A replaced buffer stays allocated: CUDA graphs captured earlier hold its address, work in flight may still use
      // it, and nothing may synchronise or free while a capture is under way.  Growth is geometric, so the retired
      // buffers of a stream add up to less than its current one.
      g_retired.push_back(s);
      s = Scratch();
    }
    if (capture != 0) {
      s.holder = at::empty({(int64_t)cap}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, dev));
      s.ptr = s.holder.data_ptr();
    } else {
      s.ptr = blr_scratch_alloc(cap);
      TORCH_CHECK(s.ptr != nullptr, "blr_b200: ", blr_last_error());
    }
    s.bytes = cap;
    s.unset = is_ws;
  }
  if (s.unset && (capture == 0 || capture != s.capture)) {
    check_rc(blr_workspace_init(s.ptr, s.bytes, st));
    s.unset = capture != 0;
    s.capture = capture;
  }
  return {s.ptr, s.bytes};
}

// Workspace of an operator call: with room for the planes of a cut contraction, which the library uses when it is given it.  Up to 16
// tokens four fp32 planes of intermediates per group (long in-blocks); one group (low rank) above: four planes, up to 64 MB.
size_t call_ws_bytes(int64_t n, int64_t groups, int64_t width) {
  const size_t base = blr_workspace_bytes(n, groups, width), inter = (size_t)groups * n * width;
  if (n <= 16) return base + (groups > 1 ? inter * 10 : 0);
  return base + (groups == 1 ? std::min(inter * 16, (size_t)64 << 20) : 0);
}

int dtype_code(const at::Tensor& x) {
  if (x.scalar_type() == at::kHalf) return BLR_DTYPE_F16;
  TORCH_CHECK(x.scalar_type() == at::kBFloat16, "expected float16 or bfloat16 tensors, got ", x.scalar_type());
  return BLR_DTYPE_BF16;
}

// (N, I) activations as the TMA rules want them: unit inner stride, row stride a multiple of 8 elements, 16-byte
// aligned base; copies only if the input forces it.
at::Tensor rows(const at::Tensor& x) {
  TORCH_CHECK(x.dim() == 2, "x must be (tokens, features)");
  at::Tensor r = x;
  if (r.stride(1) != 1 || (r.size(0) > 1 && r.stride(0) % 8 != 0) || reinterpret_cast<uintptr_t>(r.data_ptr()) % 16 != 0) {
    r = r.contiguous();
    if (reinterpret_cast<uintptr_t>(r.data_ptr()) % 16 != 0) r = r.clone();
  }
  return r;
}

void need_factors(const at::Tensor& x, std::initializer_list<const at::Tensor*> factors) {
  TORCH_CHECK(x.is_cuda(), "blr_b200 operators need CUDA tensors: there is no CPU implementation in this package");
  for (const at::Tensor* t : factors) {
    TORCH_CHECK(t->is_cuda() && t->device() == x.device(), "x and the factors must live on one CUDA device");
    TORCH_CHECK(t->is_contiguous(), "factor tensors must be contiguous");
  }
}

struct Call {
  c10::cuda::CUDAGuard guard;
  cudaStream_t st;
  int dev;
  explicit Call(const at::Tensor& x) : guard(x.device()), st(at::cuda::getCurrentCUDAStream(x.device().index()).stream()), dev(x.device().index()) {}
  Room ws(int64_t n, int64_t groups, int64_t width) { return scratch(g_ws, dev, st, call_ws_bytes(n, groups, width), true); }
};

// ----------------------------------------------------------------------------------------------- operators
at::Tensor blast(const at::Tensor& x_in, const at::Tensor& U, const at::Tensor& V, const at::Tensor& S, int64_t u_layout,
                 int64_t v_layout, int64_t s_i, int64_t s_j, int64_t s_r, int64_t b, int64_t P, int64_t Q, int64_t R, int64_t flags,
                 int64_t b_out, const c10::optional<at::Tensor>& E) {
  need_factors(x_in, {&U, &V, &S});
  const int64_t bo = b_out < 0 ? b : b_out;
  if (x_in.size(0) == 0) return at::empty({0, bo * Q}, x_in.options());
  const at::Tensor x = rows(x_in);
  TORCH_CHECK(U.scalar_type() == x.scalar_type() && V.scalar_type() == x.scalar_type() && S.scalar_type() == x.scalar_type(),
              "x, U, V, S must share one 16-bit dtype");
  Call c(x);
  const int64_t n = x.size(0);
  at::Tensor out = at::empty({n, bo * Q}, x.options());
  const Room w = c.ws(n, b, R);
  const void* e_ready = nullptr;  // expanded coupling factors built once by the caller (prefill sizes)
  if (E.has_value() && E->defined()) {
    TORCH_CHECK(E->is_cuda() && E->device() == x.device() && E->is_contiguous() &&
                    (size_t)E->nbytes() >= blr_blast_coupling_bytes((int)b, (int)bo, (int)R),
                "E must hold blr_blast_coupling_bytes bytes on x's device");
    e_ready = E->data_ptr();
  }
  check_rc(blr_blast_rows_prepared(x.data_ptr(), x.stride(0), n, dtype_code(x), U.data_ptr(), (int)u_layout, V.data_ptr(),
                                   (int)v_layout, S.data_ptr(), s_i, s_j, s_r, (int)b, (int)bo, (int)P, (int)Q, (int)R, (int)flags,
                                   out.data_ptr(), out.stride(0), w.ptr, w.bytes, c.st, e_ready));
  return out;
}

at::Tensor blast_wq(const at::Tensor& x_in, const at::Tensor& Uq, const at::Tensor& u_scale, const at::Tensor& Vq,
                    const at::Tensor& v_scale, const at::Tensor& S, int64_t s_i, int64_t s_j, int64_t s_r, int64_t bits,
                    int64_t group, int64_t b, int64_t P, int64_t Q, int64_t R) {
  need_factors(x_in, {&Uq, &u_scale, &Vq, &v_scale, &S});
  if (x_in.size(0) == 0) return at::empty({0, b * Q}, x_in.options());
  const at::Tensor x = rows(x_in);
  TORCH_CHECK(u_scale.scalar_type() == at::kHalf && v_scale.scalar_type() == at::kHalf, "scales are fp16");
  TORCH_CHECK(S.scalar_type() == x.scalar_type(), "x and S must share one 16-bit dtype");
  Call c(x);
  const int64_t n = x.size(0);
  at::Tensor out = at::empty({n, b * Q}, x.options());
  const Room w = c.ws(n, b, R);
  check_rc(blr_blast_wq(x.data_ptr(), x.stride(0), n, dtype_code(x), Uq.data_ptr(), u_scale.data_ptr(), Vq.data_ptr(),
                        v_scale.data_ptr(), S.data_ptr(), s_i, s_j, s_r, (int)bits, (int)group, (int)b, (int)P, (int)Q, (int)R,
                        out.data_ptr(), out.stride(0), w.ptr, w.bytes, c.st));
  return out;
}

at::Tensor monarch(const at::Tensor& x_in, const at::Tensor& w1, const at::Tensor& w2, int64_t w1_layout, int64_t w1_cols,
                   int64_t w2_layout, int64_t b, int64_t P, int64_t rank, int64_t Qs, int64_t out_order) {
  need_factors(x_in, {&w1, &w2});
  if (x_in.size(0) == 0) return at::empty({0, b * Qs}, x_in.options());
  const at::Tensor x = rows(x_in);
  TORCH_CHECK(w1.scalar_type() == x.scalar_type() && w2.scalar_type() == x.scalar_type(), "x and the factors must share one 16-bit dtype");
  Call c(x);
  const int64_t n = x.size(0);
  at::Tensor out = at::empty({n, b * Qs}, x.options());
  const Room w = c.ws(n, b, rank);
  check_rc(blr_monarch(x.data_ptr(), x.stride(0), n, dtype_code(x), w1.data_ptr(), (int)w1_layout, (int)w1_cols, w2.data_ptr(),
                       (int)w2_layout, (int)b, (int)P, (int)rank, (int)Qs, (int)out_order, out.data_ptr(), out.stride(0), w.ptr,
                       w.bytes, c.st));
  return out;
}

at::Tensor low_rank(const at::Tensor& x_in, const at::Tensor& V, const at::Tensor& U, int64_t v_layout, int64_t u_layout, int64_t I,
                    int64_t R, int64_t O) {
  need_factors(x_in, {&V, &U});
  if (x_in.size(0) == 0) return at::empty({0, O}, x_in.options());
  const at::Tensor x = rows(x_in);
  TORCH_CHECK(V.scalar_type() == x.scalar_type() && U.scalar_type() == x.scalar_type(), "x and the factors must share one 16-bit dtype");
  Call c(x);
  const int64_t n = x.size(0);
  at::Tensor out = at::empty({n, O}, x.options());
  const Room w = c.ws(n, 1, R);
  check_rc(blr_low_rank(x.data_ptr(), x.stride(0), n, dtype_code(x), V.data_ptr(), (int)v_layout, U.data_ptr(), (int)u_layout, (int)I,
                        (int)R, (int)O, out.data_ptr(), out.stride(0), w.ptr, w.bytes, c.st));
  return out;
}

at::Tensor dense(const at::Tensor& x_in, const at::Tensor& W, int64_t w_layout, int64_t I, int64_t O) {
  need_factors(x_in, {&W});
  if (x_in.size(0) == 0) return at::empty({0, O}, x_in.options());
  const at::Tensor x = rows(x_in);
  TORCH_CHECK(W.scalar_type() == x.scalar_type(), "x and W must share one 16-bit dtype");
  Call c(x);
  const int64_t n = x.size(0);
  at::Tensor out = at::empty({n, O}, x.options());
  check_rc(blr_dense(x.data_ptr(), x.stride(0), n, dtype_code(x), W.data_ptr(), (int)w_layout, (int)I, (int)O, out.data_ptr(),
                     out.stride(0), c.st));
  return out;
}

// Host-buffer call (x_host and out_host pinned, N <= 16): copy-in, kernels and copy-out of consecutive calls overlap on
// the library's copy streams; out_host is valid after host_flush() and a synchronisation of the current stream.
void blast_wq_host(const at::Tensor& x_host, at::Tensor& out_host, const at::Tensor& Uq, const at::Tensor& u_scale,
                   const at::Tensor& Vq, const at::Tensor& v_scale, const at::Tensor& S, int64_t bits, int64_t group) {
  TORCH_CHECK(!x_host.is_cuda() && !out_host.is_cuda(), "x_host and out_host are host tensors");
  need_factors(S, {&Uq, &u_scale, &Vq, &v_scale});
  const int64_t per = bits == 8 ? 1 : 2;
  const int64_t b = u_scale.size(0), Q = u_scale.size(1), R = v_scale.size(1), P = Vq.size(-1) * per, n = x_host.size(0);
  TORCH_CHECK(x_host.dim() == 2 && out_host.dim() == 2 && n <= 16 && x_host.size(1) == b * P && out_host.size(0) == n &&
                  out_host.size(1) == b * Q && x_host.scalar_type() == S.scalar_type() && out_host.scalar_type() == S.scalar_type() &&
                  x_host.stride(1) == 1 && out_host.stride(1) == 1,
              "x_host (N <= 16, b*P) and out_host (N, b*Q) must be 16-bit host tensors of the factors' dtype");
  Call c(S);
  const Room w = scratch(g_ws, c.dev, c.st, blr_workspace_bytes(16, b, R), true);
  const Room sg = scratch(g_staging, c.dev, c.st, blr_host_staging_bytes(16, b * P, b * Q), false);
  check_rc(blr_blast_wq_host(x_host.data_ptr(), x_host.stride(0), n, dtype_code(S), Uq.data_ptr(), u_scale.data_ptr(), Vq.data_ptr(),
                             v_scale.data_ptr(), S.data_ptr(), b * R, R, 1, (int)bits, (int)group, (int)b, (int)P, (int)Q, (int)R,
                             out_host.data_ptr(), out_host.stride(0), sg.ptr, sg.bytes, w.ptr, w.bytes, c.st));
}

void host_flush(int64_t device) {
  c10::cuda::CUDAGuard guard((c10::DeviceIndex)device);
  check_rc(blr_host_flush(at::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream()));
}

// The workspace of (device, stream), grown to at least nbytes: (pointer, bytes).  For the parts of the Python layer that
// still call the C ABI through ctypes, and for tests that look into the scratch.
std::vector<int64_t> workspace(int64_t device, int64_t stream, int64_t nbytes) {
  c10::cuda::CUDAGuard guard((c10::DeviceIndex)device);
  const Room w = scratch(g_ws, (int)device, reinterpret_cast<cudaStream_t>(stream), (size_t)nbytes, true);
  return {(int64_t)reinterpret_cast<uintptr_t>(w.ptr), (int64_t)w.bytes};
}

// The staging buffer of the host-buffer calls of (device, stream), likewise.
std::vector<int64_t> staging(int64_t device, int64_t stream, int64_t nbytes) {
  c10::cuda::CUDAGuard guard((c10::DeviceIndex)device);
  const Room w = scratch(g_staging, (int)device, reinterpret_cast<cudaStream_t>(stream), (size_t)nbytes, false);
  return {(int64_t)reinterpret_cast<uintptr_t>(w.ptr), (int64_t)w.bytes};
}

// Status of the workspace of (device, stream) (synchronises the stream): 0, or a BLR_ERR_* code after which the
// workspace has been re-initialised.
int64_t workspace_status(int64_t device, int64_t stream) {
  c10::cuda::CUDAGuard guard((c10::DeviceIndex)device);
  Scratch s;
  {
    std::lock_guard<std::mutex> lock(g_mu);
    auto it = g_ws.find({(int)device, reinterpret_cast<cudaStream_t>(stream)});
    if (it == g_ws.end()) return 0;
    s = it->second;
  }
  const int rc = blr_workspace_status(s.ptr, reinterpret_cast<void*>(stream));
  if (rc != 0) blr_workspace_init(s.ptr, s.bytes, reinterpret_cast<void*>(stream));
  return rc;
}

// ----------------------------------------------------------------------------------------------- shapes only
at::Tensor blast_meta(const at::Tensor& x, const at::Tensor&, const at::Tensor&, const at::Tensor&, int64_t, int64_t, int64_t, int64_t,
                      int64_t, int64_t b, int64_t, int64_t Q, int64_t, int64_t, int64_t b_out, const c10::optional<at::Tensor>&) {
  return at::empty_symint({x.sym_size(0), c10::SymInt((b_out < 0 ? b : b_out) * Q)}, x.options());
}
at::Tensor blast_wq_meta(const at::Tensor& x, const at::Tensor&, const at::Tensor&, const at::Tensor&, const at::Tensor&,
                         const at::Tensor&, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t b, int64_t, int64_t Q, int64_t) {
  return at::empty_symint({x.sym_size(0), c10::SymInt(b * Q)}, x.options());
}
at::Tensor monarch_meta(const at::Tensor& x, const at::Tensor&, const at::Tensor&, int64_t, int64_t, int64_t, int64_t b, int64_t, int64_t,
                        int64_t Qs, int64_t) {
  return at::empty_symint({x.sym_size(0), c10::SymInt(b * Qs)}, x.options());
}
at::Tensor low_rank_meta(const at::Tensor& x, const at::Tensor&, const at::Tensor&, int64_t, int64_t, int64_t, int64_t, int64_t O) {
  return at::empty_symint({x.sym_size(0), c10::SymInt(O)}, x.options());
}
at::Tensor dense_meta(const at::Tensor& x, const at::Tensor&, int64_t, int64_t, int64_t O) {
  return at::empty_symint({x.sym_size(0), c10::SymInt(O)}, x.options());
}

}  // namespace

TORCH_LIBRARY(blr_b200_ext, m) {
  m.def("blast(Tensor x, Tensor U, Tensor V, Tensor S, int u_layout, int v_layout, int s_i, int s_j, int s_r, int b, int P, int Q, "
        "int R, int flags, int b_out=-1, Tensor? E=None) -> Tensor");
  m.def("blast_wq(Tensor x, Tensor Uq, Tensor u_scale, Tensor Vq, Tensor v_scale, Tensor S, int s_i, int s_j, int s_r, int bits, "
        "int group, int b, int P, int Q, int R) -> Tensor");
  m.def("monarch(Tensor x, Tensor w1, Tensor w2, int w1_layout, int w1_cols, int w2_layout, int b, int P, int rank, int Qs, "
        "int out_order) -> Tensor");
  m.def("low_rank(Tensor x, Tensor V, Tensor U, int v_layout, int u_layout, int I, int R, int O) -> Tensor");
  m.def("dense(Tensor x, Tensor W, int w_layout, int I, int O) -> Tensor");
  m.def("blast_wq_host(Tensor x_host, Tensor(a!) out_host, Tensor Uq, Tensor u_scale, Tensor Vq, Tensor v_scale, Tensor S, int bits, "
        "int group) -> ()");
  m.def("host_flush(int device) -> ()", &host_flush);
  m.def("workspace(int device, int stream, int nbytes) -> int[]", &workspace);
  m.def("staging(int device, int stream, int nbytes) -> int[]", &staging);
  m.def("workspace_status(int device, int stream) -> int", &workspace_status);
}

TORCH_LIBRARY_IMPL(blr_b200_ext, CUDA, m) {
  m.impl("blast", &blast);
  m.impl("blast_wq", &blast_wq);
  m.impl("monarch", &monarch);
  m.impl("low_rank", &low_rank);
  m.impl("dense", &dense);
}

// CPU tensors: the same refusal as everywhere else in this package (the device functions check is_cuda first)
TORCH_LIBRARY_IMPL(blr_b200_ext, CPU, m) {
  m.impl("blast", &blast);
  m.impl("blast_wq", &blast_wq);
  m.impl("monarch", &monarch);
  m.impl("low_rank", &low_rank);
  m.impl("dense", &dense);
}

// the host-buffer call mixes host tensors (x, out) with device tensors (factors): one kernel for every backend key
TORCH_LIBRARY_IMPL(blr_b200_ext, CompositeExplicitAutograd, m) { m.impl("blast_wq_host", &blast_wq_host); }

TORCH_LIBRARY_IMPL(blr_b200_ext, Meta, m) {
  m.impl("blast", &blast_meta);
  m.impl("blast_wq", &blast_wq_meta);
  m.impl("monarch", &monarch_meta);
  m.impl("low_rank", &low_rank_meta);
  m.impl("dense", &dense_meta);
}

// ----------------------------------------------------------------------------------------------- direct calls
// The eager route of the Python layer.  An operator call through torch.ops costs the host 14 - 21 us (4.6 - 8.5 here) - argument parsing
// against the schema, the boxed dispatcher hop, one more for the output's allocation, and the shape checks in Python ahead
// of it - which is more than the kernels of a decode-size call take.  These functions take the Python layer's own arguments,
// check them, allocate the output (leading dimensions included) and make the library call.  Whatever is not the plain case
// (tensor subclasses, a mode, a tracer or a function transform, a call that autograd records, an empty batch, a layout that needs a copy, arguments that do not fit)
// returns None and goes the general way, which also raises the errors.
namespace {

// The dispatcher would go straight to the CUDA kernel: beside the backend's key only those of the autograd bookkeeping and of autocast,
// which have nothing to do for these operators.  Anything else, on the tensor or on the thread (the tracer of torch.jit.trace, a batched
// tensor of torch.vmap or torch.func, functionalisation, a negated view), has to see the operator.
bool plain_keys(const at::Tensor& t) {
  static const uint64_t allowed = (c10::DispatchKeySet({c10::DispatchKey::CUDA, c10::DispatchKey::BackendSelect, c10::DispatchKey::ADInplaceOrView}) |
                                   c10::autograd_dispatch_keyset | c10::autocast_dispatch_keyset).raw_repr();
  const auto tls = c10::impl::tls_local_dispatch_key_set();
  return (((t.key_set() | tls.included_) - tls.excluded_).raw_repr() & ~allowed) == 0;
}

const at::Tensor* plain(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  return plain_keys(t) ? &t : nullptr;
}

struct Direct {
  int dev = -1;
  at::ScalarType dt = at::kHalf;
  int64_t n = 0, width = 0, ldx = 0;
  const at::Tensor* x = nullptr;
  cudaStream_t st = nullptr;

  // x: (..., width) CUDA tensor of a 16-bit type on the current device, whose rows the kernels can read as they lie
  bool take_x(PyObject* o) {
    x = plain(o);
    if (x == nullptr || c10::impl::dispatch_mode_enabled() || at::impl::torch_function_mode_enabled() || !x->is_cuda()) return false;
    dt = x->scalar_type();
    const int64_t dim = x->dim();
    if ((dt != at::kHalf && dt != at::kBFloat16) || dim < 2) return false;
    const at::IntArrayRef sz = x->sizes(), sd = x->strides();
    width = sz[dim - 1];
    if (dim == 2) {
      n = sz[0];
      ldx = sd[0];
      if (sd[1] != 1 || (n > 1 && ldx % 8 != 0)) return false;
      if (n == 1) {  // the stride of a single row means nothing
        if (width % 8 != 0) return false;
        ldx = width;
      }
    } else {
      if (!x->is_contiguous() || width % 8 != 0) return false;
      n = x->numel() / (width > 0 ? width : 1);
      ldx = width;
    }
    if (n == 0 || width == 0 || reinterpret_cast<uintptr_t>(x->data_ptr()) % 16 != 0) return false;
    dev = x->device().index();
    if (dev != c10::cuda::current_device()) return false;
    st = at::cuda::getCurrentCUDAStream(dev).stream();
    return true;
  }
  // a factor of the layer: contiguous, on x's device
  const at::Tensor* factor(PyObject* o, at::ScalarType type) const {
    const at::Tensor* t = plain(o);
    return t != nullptr && t->is_cuda() && t->device().index() == dev && t->scalar_type() == type && t->is_contiguous() ? t : nullptr;
  }
  int code() const { return dt == at::kHalf ? BLR_DTYPE_F16 : BLR_DTYPE_BF16; }
  // (..., O) with x's leading dimensions, or (N, O)
  at::Tensor output(int64_t O, bool keep_dims = true) const {
    if (x->dim() == 2 || !keep_dims) return at::detail::empty_cuda({n, O}, dt, x->device(), c10::nullopt);
    c10::SmallVector<int64_t, 6> sz(x->sizes().begin(), x->sizes().end());
    sz.back() = O;
    return at::detail::empty_cuda(sz, dt, x->device(), c10::nullopt);
  }
  // the stream's workspace
  Room ws(int64_t groups, int64_t w, size_t at_least = 0) const {
    size_t need = call_ws_bytes(n, groups, w);
    if (need < at_least) need = at_least;
    return scratch(g_ws, dev, st, need, true);
  }
};

#define BLR_NONE() do { Py_RETURN_NONE; } while (0)

// Whether autograd would record the call: the dispatcher then gives the result a node that says, in a backward pass, that the operator has
// no derivative.  A result without it would end the gradient's way silently.
bool records_grad(std::initializer_list<const at::Tensor*> ts) {
  if (!at::GradMode::is_enabled()) return false;
  for (const at::Tensor* t : ts)
    if (t->requires_grad()) return true;
  return false;
}

// The rest of the function under the operator's name in a profile, as the dispatcher records it (nothing without a profiler)
#define BLR_RECORD(op, ...) RECORD_FUNCTION("blr_b200_ext::" op, (std::vector<c10::IValue>{__VA_ARGS__}))

// n integer arguments; false, with no Python error left behind, when one of them is none
bool take_ints(PyObject* const* a, int n, long* v) {
  for (int i = 0; i < n; ++i) {
    v[i] = PyLong_AsLong(a[i]);
    if (v[i] == -1 && PyErr_Occurred()) {
      PyErr_Clear();
      return false;
    }
  }
  return true;
}

// Python's lock is free for the rest of the scope: a launch blocks when the stream's queue is full, and the registry of workspaces, which
// allocates under its own lock, must not be waited for with Python's (an allocation that torch records a stack for wants that).
struct NoGil {
  PyThreadState* state = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(state); }
};

template <typename F>
void call_library(F&& f) {
  int rc;
  {
    NoGil free;
    rc = f();
  }
  check_rc(rc);
}

// blast(x, U, V, S, family, flags, e_tokens, e_blocks, e_rank): above e_tokens tokens layers of at most e_blocks blocks and e_rank
// ranks are left to the Python layer, which keeps prepared coupling factors for them.  family 0 torch layouts U (b,Q,R), V (b,R,P), S (b,b,R); 1 U (b,R,Q), V (b,P,R),
// S (b_in,b_out,R); 2 U (b,Q,R), V (b,P,R), S (R,b_out,b_in).
PyObject* py_blast(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  Direct d;
  long v_int[5];
  if (na != 9 || !d.take_x(a[0]) || !take_ints(a + 4, 5, v_int)) BLR_NONE();
  const at::Tensor *U = d.factor(a[1], d.dt), *V = d.factor(a[2], d.dt), *S = d.factor(a[3], d.dt);
  const long family = v_int[0], flags = v_int[1];
  if (!U || !V || !S || U->dim() != 3 || V->dim() != 3 || S->dim() != 3) BLR_NONE();
  const at::IntArrayRef u = U->sizes(), v = V->sizes(), s = S->sizes();
  const int64_t b = v[0], R = family == 0 ? v[1] : v[2], P = family == 0 ? v[2] : v[1], Q = family == 1 ? u[2] : u[1];
  if (b < 2 || u[0] != b || (family == 1 ? u[1] : u[2]) != R || d.width != b * P) BLR_NONE();
  if (d.n > v_int[2] && b <= v_int[3] && R <= v_int[4]) BLR_NONE();
  int64_t si, sj, sr;
  if (family == 2) {
    if (s[0] != R || s[1] != b || s[2] != b) BLR_NONE();
    si = b, sj = 1, sr = b * b;
  } else {
    if (s[0] != b || s[1] != b || s[2] != R) BLR_NONE();
    si = family == 0 ? b * R : R, sj = family == 0 ? R : b * R, sr = 1;
  }
  if (records_grad({d.x, U, V, S})) BLR_NONE();
  BLR_RECORD("blast", *d.x, *U, *V, *S);
  at::Tensor out = d.output(b * Q);
  void* o = out.data_ptr();
  call_library([&] {
    const Room w = d.ws(b, R);
    return blr_blast(d.x->data_ptr(), d.ldx, d.n, d.code(), U->data_ptr(), family == 1 ? BLR_W_MMAJOR : BLR_W_KMAJOR, V->data_ptr(),
                     family == 0 ? BLR_W_KMAJOR : BLR_W_MMAJOR, S->data_ptr(), si, sj, sr, (int)b, (int)P, (int)Q, (int)R, (int)flags, o,
                     b * Q, w.ptr, w.bytes, d.st);
  });
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// Shapes of a weight-quantised layer (Uq, u_scale, Vq, v_scale, S); false: not what the call expects.
struct QuantLayer {
  const at::Tensor *Uq, *us, *Vq, *vs, *S;
  int64_t b, P, Q, R;
  bool take(const Direct& d, PyObject* const* a, long bits, long group) {
    const at::ScalarType qt = bits == 8 ? at::kChar : at::kByte;
    Uq = d.factor(a[0], qt), us = d.factor(a[1], at::kHalf), Vq = d.factor(a[2], qt), vs = d.factor(a[3], at::kHalf), S = d.factor(a[4], d.dt);
    const int64_t dim = group == 0 ? 2 : 3, per = bits == 8 ? 1 : 2;
    if (!Uq || !us || !Vq || !vs || !S || Uq->dim() != 3 || Vq->dim() != 3 || S->dim() != 3 || us->dim() != dim || vs->dim() != dim) return false;
    const at::IntArrayRef u = Uq->sizes(), v = Vq->sizes(), s = S->sizes(), a_us = us->sizes(), a_vs = vs->sizes();
    b = a_us[0], Q = a_us[1], R = a_vs[1], P = v[2] * per;
    if (b < 2 || a_vs[0] != b || u[0] != b || u[1] != Q || u[2] * per != R || v[0] != b || v[1] != R || s[0] != b || s[1] != b || s[2] != R) return false;
    if (group != 0 && (a_us[2] * group != R || a_vs[2] * group != P)) return false;
    return true;
  }
};

// Layers that take twice as many tokens before their factors are widened in a pass (WQ_LARGE_LAYER)
bool large_layer(int64_t b, int64_t P, int64_t Q, int64_t R) { return b * R * (P + Q) >= (1 << 20); }

// blast_wq(x, Uq, u_scale, Vq, v_scale, S, bits, group, max_tokens): beyond max_tokens, twice that for a large layer, it is the Python layer's
PyObject* py_blast_wq(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  Direct d;
  long v_int[3];
  if (na != 9 || !d.take_x(a[0]) || !take_ints(a + 6, 3, v_int)) BLR_NONE();
  const long bits = v_int[0], group = v_int[1];
  QuantLayer q;
  if ((bits != 8 && bits != 4) || d.n > 2 * v_int[2] || !q.take(d, a + 1, bits, group) || d.width != q.b * q.P) BLR_NONE();
  if (d.n > v_int[2] * (large_layer(q.b, q.P, q.Q, q.R) ? 2 : 1)) BLR_NONE();
  if (d.n > 16 && ((q.P * bits / 8) % 16 != 0 || (q.R * bits / 8) % 16 != 0)) BLR_NONE();
  if (records_grad({d.x, q.us, q.vs, q.S})) BLR_NONE();
  BLR_RECORD("blast_wq", *d.x, *q.Uq, *q.us, *q.Vq, *q.vs, *q.S);
  at::Tensor out = d.output(q.b * q.Q);
  void* o = out.data_ptr();
  call_library([&] {
    const Room w = d.ws(q.b, q.R);
    return blr_blast_wq(d.x->data_ptr(), d.ldx, d.n, d.code(), q.Uq->data_ptr(), q.us->data_ptr(), q.Vq->data_ptr(), q.vs->data_ptr(),
                        q.S->data_ptr(), q.b * q.R, q.R, 1, (int)bits, (int)group, (int)q.b, (int)q.P, (int)q.Q, (int)q.R, o, q.b * q.Q,
                        w.ptr, w.bytes, d.st);
  });
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// monarch(x, w1, w2, w1_mmajor, w2_mmajor, interleaved): w1 (b,P,rank) with grouped columns or, K-major, (b,rank,P) in the torch
// order; w2 (b,Q,rank) or, M-major, (b,rank,Q).
PyObject* py_monarch(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  Direct d;
  long v_int[3];
  if (na != 6 || !d.take_x(a[0]) || !take_ints(a + 3, 3, v_int)) BLR_NONE();
  const at::Tensor *w1 = d.factor(a[1], d.dt), *w2 = d.factor(a[2], d.dt);
  const bool m1 = v_int[0] != 0, m2 = v_int[1] != 0, inter = v_int[2] != 0;
  if (!w1 || !w2 || w1->dim() != 3 || w2->dim() != 3) BLR_NONE();
  const at::IntArrayRef p = w1->sizes(), q = w2->sizes();
  const int64_t b = p[0], P = m1 ? p[1] : p[2], rank = m1 ? p[2] : p[1], Q = m2 ? q[2] : q[1];
  if (b < 1 || q[0] != b || (m2 ? q[1] : q[2]) != rank || rank % b != 0 || d.width != b * P) BLR_NONE();
  if (records_grad({d.x, w1, w2})) BLR_NONE();
  BLR_RECORD("monarch", *d.x, *w1, *w2);
  at::Tensor out = d.output(b * Q);
  void* o = out.data_ptr();
  call_library([&] {
    const Room w = d.ws(b, rank);
    return blr_monarch(d.x->data_ptr(), d.ldx, d.n, d.code(), w1->data_ptr(), m1 ? BLR_W_MMAJOR : BLR_W_KMAJOR,
                       m1 ? BLR_MONARCH_COLS_GROUPED : BLR_MONARCH_COLS_TORCH, w2->data_ptr(), m2 ? BLR_W_MMAJOR : BLR_W_KMAJOR, (int)b, (int)P,
                       (int)rank, (int)Q, inter ? BLR_OUT_INTERLEAVED : BLR_OUT_BLOCKED, o, b * Q, w.ptr, w.bytes, d.st);
  });
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// low_rank(x, V, U, mmajor): V (I,R), U (R,O), result (N,O); K-major: V (R,I), U (O,R), x's leading dimensions kept.
PyObject* py_low_rank(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  Direct d;
  long v_int;
  if (na != 4 || !d.take_x(a[0]) || !take_ints(a + 3, 1, &v_int)) BLR_NONE();
  const at::Tensor *V = d.factor(a[1], d.dt), *U = d.factor(a[2], d.dt);
  const bool m = v_int != 0;
  if (!V || !U || V->dim() != 2 || U->dim() != 2) BLR_NONE();
  const int64_t I = V->size(m ? 0 : 1), R = V->size(m ? 1 : 0), O = U->size(m ? 1 : 0);
  if (U->size(m ? 0 : 1) != R || d.width != I || R == 0 || O == 0) BLR_NONE();
  if (records_grad({d.x, V, U})) BLR_NONE();
  BLR_RECORD("low_rank", *d.x, *V, *U);
  at::Tensor out = d.output(O, !m);
  void* o = out.data_ptr();
  const int layout = m ? BLR_W_MMAJOR : BLR_W_KMAJOR;
  call_library([&] {
    const Room w = d.ws(1, R);
    return blr_low_rank(d.x->data_ptr(), d.ldx, d.n, d.code(), V->data_ptr(), layout, U->data_ptr(), layout, (int)I, (int)R, (int)O, o, O,
                        w.ptr, w.bytes, d.st);
  });
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// dense(x, W, mmajor): W (I,O), result (N,O); K-major: W (O,I), x's leading dimensions kept.
PyObject* py_dense(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  Direct d;
  long v_int;
  if (na != 3 || !d.take_x(a[0]) || !take_ints(a + 2, 1, &v_int)) BLR_NONE();
  const at::Tensor* W = d.factor(a[1], d.dt);
  const bool m = v_int != 0;
  if (!W || W->dim() != 2) BLR_NONE();
  const int64_t I = W->size(m ? 0 : 1), O = W->size(m ? 1 : 0);
  if (d.width != I || O == 0) BLR_NONE();
  if (records_grad({d.x, W})) BLR_NONE();
  BLR_RECORD("dense", *d.x, *W);
  at::Tensor out = d.output(O, !m);
  void* o = out.data_ptr();
  call_library([&] {
    return blr_dense(d.x->data_ptr(), d.ldx, d.n, d.code(), W->data_ptr(), m ? BLR_W_MMAJOR : BLR_W_KMAJOR, (int)I, (int)O, o, O, d.st);
  });
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// multi(x, layers, bits, group, x_mul, biases, residuals, out_act): the fused call for layers of equal shape on one input
// (blr_blast_multi); layers: list of (U, Vt, S) or (Uq, u_scale, Vq, v_scale, S).  Returns the list of outputs, or None where the call
// does not apply (see blast_multi in ops.py for the token counts).
PyObject* py_multi(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  Direct d;
  long v_int[2], out_act;
  if (na != 8 || !PyList_CheckExact(a[1]) || !d.take_x(a[0]) || !take_ints(a + 2, 2, v_int) || !take_ints(a + 7, 1, &out_act)) BLR_NONE();
  const Py_ssize_t k = PyList_GET_SIZE(a[1]);
  const long bits = v_int[0], group = v_int[1];
  if (k < 1 || k > 3 || (out_act != 0 && d.n <= 16)) BLR_NONE();
  const at::Tensor* xm = nullptr;
  if (a[4] != Py_None) {
    xm = plain(a[4]);
    if (!xm || !xm->is_cuda() || xm->scalar_type() != d.dt || xm->sizes() != d.x->sizes() || xm->strides() != d.x->strides() ||
        reinterpret_cast<uintptr_t>(xm->data_ptr()) % 16 != 0)
      BLR_NONE();
  }
  blr_blast_problem pr[3] = {};
  int64_t b = 0, P = 0, Q = 0, R = 0;
  bool any_bias = false, any_res = false;
  for (Py_ssize_t i = 0; i < k; ++i) {
    PyObject* lay = PyList_GET_ITEM(a[1], i);
    if (!PyTuple_CheckExact(lay) || PyTuple_GET_SIZE(lay) != (bits == 16 ? 3 : 5)) BLR_NONE();
    int64_t b1, P1, Q1, R1;
    if (bits == 16) {
      const at::Tensor *U = d.factor(PyTuple_GET_ITEM(lay, 0), d.dt), *V = d.factor(PyTuple_GET_ITEM(lay, 1), d.dt),
                       *S = d.factor(PyTuple_GET_ITEM(lay, 2), d.dt);
      if (!U || !V || !S || U->dim() != 3 || V->dim() != 3 || S->dim() != 3) BLR_NONE();
      b1 = V->size(0), R1 = V->size(1), P1 = V->size(2), Q1 = U->size(1);
      if (U->size(0) != b1 || U->size(2) != R1 || S->size(0) != b1 || S->size(1) != b1 || S->size(2) != R1) BLR_NONE();
      pr[i].U = U->data_ptr(), pr[i].V = V->data_ptr(), pr[i].S = S->data_ptr();
    } else {
      QuantLayer q;
      PyObject* items[5];
      for (int j = 0; j < 5; ++j) items[j] = PyTuple_GET_ITEM(lay, j);
      if ((bits != 8 && bits != 4) || !q.take(d, items, bits, group)) BLR_NONE();
      b1 = q.b, P1 = q.P, Q1 = q.Q, R1 = q.R;
      pr[i].U = q.Uq->data_ptr(), pr[i].V = q.Vq->data_ptr(), pr[i].S = q.S->data_ptr();
      pr[i].u_scale = q.us->data_ptr(), pr[i].v_scale = q.vs->data_ptr();
    }
    if (i == 0) b = b1, P = P1, Q = Q1, R = R1;
    else if (b != b1 || P != P1 || Q != Q1 || R != R1) BLR_NONE();
    for (int which = 0; which < 2; ++which) {
      PyObject* list = a[5 + which];
      if (list == Py_None) continue;
      if (!PyList_CheckExact(list) || PyList_GET_SIZE(list) != k) BLR_NONE();
      PyObject* item = PyList_GET_ITEM(list, i);
      if (item == Py_None) continue;
      const at::Tensor* t = d.factor(item, d.dt);
      if (!t || t->numel() != (which == 0 ? b * Q : d.n * b * Q) || (which == 1 && reinterpret_cast<uintptr_t>(t->data_ptr()) % 16 != 0)) BLR_NONE();
      if (which == 0) pr[i].bias = t->data_ptr(), any_bias = true;
      else pr[i].residual = t->data_ptr(), pr[i].ldr = b * Q, any_res = true;
    }
  }
  if (b < 2 || d.width != b * P) BLR_NONE();
  const bool prefill = d.n > 16 && !xm && (any_bias || any_res || out_act != 0) && !(any_res && (d.n <= 64 || d.n > 512));
  // (heavy layers stay ahead of separate calls up to 16 tokens: two of 4096 -> 11008, R = 1488, 16 tokens 48.5 -> 40.8 us; three of the heaviest
  // while the planes are few: 4096 -> 11008, R = 1488, 8 / 10 / 16 tokens 59.0 | 70.6 | 72.8 separate, 51.1 | 72.3 | 81.3 fused; R = 1024, 12 /
  // 16 tokens 58.5 | 51.6, 54.8 | 52.7)
  const bool heavy = bits == 16 && k > 1 && 2ll * b * R * (P + Q) >= (12ll << 20) &&
                     !(k == 3 && 2ll * b * R * (P + Q) >= (24ll << 20) && b * d.n * R > 200000);
  if (d.n > (heavy ? 16 : bits == 16 ? 8 : 4) && !prefill) BLR_NONE();
  if (prefill && bits != 16 && ((P * bits / 8) % 16 != 0 || (R * bits / 8) % 16 != 0 || d.n > 512 * (large_layer(b, P, Q, R) ? 2 : 1))) BLR_NONE();  // (WQ_IN_GEMM_MAX_TOKENS)
  at::Tensor outs[3];
  for (Py_ssize_t i = 0; i < k; ++i) {
    outs[i] = d.output(b * Q);
    pr[i].out = outs[i].data_ptr();
    pr[i].ldo = b * Q;
  }
  int rc;
  {
    NoGil free;
    const Room w = d.ws(k * b, R, prefill ? blr_workspace_bytes(d.n, b, R) : 0);
    rc = blr_blast_multi(d.x->data_ptr(), d.ldx, xm ? xm->data_ptr() : nullptr, (xm ? BLR_ACT_SILU_MUL : BLR_ACT_NONE) | (int)out_act, d.n, d.code(),
                         (int)k, pr, b * R, R, 1, (int)bits, (int)group, (int)b, (int)P, (int)Q, (int)R, w.ptr, w.bytes, d.st);
  }
  if (rc == BLR_ERR_UNSUPPORTED) BLR_NONE();
  check_rc(rc);
  PyObject* list = PyList_New(k);
  if (list == nullptr) return nullptr;
  for (Py_ssize_t i = 0; i < k; ++i) PyList_SET_ITEM(list, i, THPVariable_Wrap(std::move(outs[i])));
  return list;
  END_HANDLE_TH_ERRORS
}

// A (d,) parameter of a norm, or None: false when it is neither.
bool norm_param(const Direct& d, PyObject* o, const void** p) {
  *p = nullptr;
  if (o == Py_None) return true;
  const at::Tensor* t = d.factor(o, d.dt);
  if (!t || t->numel() != d.width || reinterpret_cast<uintptr_t>(t->data_ptr()) % 16 != 0) return false;
  *p = t->data_ptr();
  return true;
}

// The eps of a norm; false, with no Python error left behind, when it is not a number.
bool take_eps(PyObject* o, float* eps) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1. && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  *eps = (float)v;
  return true;
}

// rmsnorm(x, weight, eps)
PyObject* py_rmsnorm(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  Direct d;
  const void* w;
  float eps;
  if (na != 3 || !d.take_x(a[0]) || !norm_param(d, a[1], &w) || w == nullptr || !take_eps(a[2], &eps)) BLR_NONE();
  at::Tensor out = d.output(d.width);
  void* o = out.data_ptr();
  call_library([&] { return blr_rmsnorm(d.x->data_ptr(), d.ldx, d.n, (int)d.width, w, eps, d.code(), o, d.width, d.st); });
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// layernorm(x, weight | None, bias | None, eps)
PyObject* py_layernorm(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  Direct d;
  const void *w, *b;
  float eps;
  if (na != 4 || !d.take_x(a[0]) || !norm_param(d, a[1], &w) || !norm_param(d, a[2], &b) || !take_eps(a[3], &eps)) BLR_NONE();
  at::Tensor out = d.output(d.width);
  void* o = out.data_ptr();
  call_library([&] {
    return blr_layernorm(d.x->data_ptr(), d.ldx, d.n, (int)d.width, w, b, eps, d.code(), o, d.width, 0, 0, 0, 0, d.st);
  });
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// add_layernorm(x, y, weight | None, bias | None, eps) -> (x + y, its norm)
PyObject* py_add_layernorm(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  Direct d;
  const void *w, *b;
  float eps;
  if (na != 5 || !d.take_x(a[0]) || !norm_param(d, a[2], &w) || !norm_param(d, a[3], &b) || !take_eps(a[4], &eps)) BLR_NONE();
  const at::Tensor* y = d.factor(a[1], d.dt);
  if (!y || y->sizes() != d.x->sizes() || reinterpret_cast<uintptr_t>(y->data_ptr()) % 16 != 0 || records_grad({d.x, y})) BLR_NONE();
  at::Tensor sum = d.output(d.width), out = d.output(d.width);
  void *s = sum.data_ptr(), *o = out.data_ptr();
  call_library([&] {
    return blr_add_layernorm(d.x->data_ptr(), d.ldx, y->data_ptr(), d.width, nullptr, 0, s, d.width, d.n, (int)d.width, w, b, eps, d.code(), o,
                             d.width, 0, 0, 0, 0, d.st);
  });
  PyObject* t = PyTuple_New(2);
  if (t == nullptr) return nullptr;
  PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(std::move(sum)));
  PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(std::move(out)));
  return t;
  END_HANDLE_TH_ERRORS
}

// A BLAST layer on 16-bit factors in the torch layouts, as the tuple (U, Vt, S, bias | None), on rows of `width` values.
struct Layer16 {
  blr_blast_problem pr = {};
  int64_t b = 0, P = 0, Q = 0, R = 0;
  bool take(const Direct& d, PyObject* o, int64_t width) {
    if (!PyTuple_CheckExact(o) || PyTuple_GET_SIZE(o) != 4) return false;
    const at::Tensor *U = d.factor(PyTuple_GET_ITEM(o, 0), d.dt), *V = d.factor(PyTuple_GET_ITEM(o, 1), d.dt), *S = d.factor(PyTuple_GET_ITEM(o, 2), d.dt);
    if (!U || !V || !S || U->dim() != 3 || V->dim() != 3 || S->dim() != 3 || records_grad({U, V, S})) return false;
    b = V->size(0), R = V->size(1), P = V->size(2), Q = U->size(1);
    if (b < 2 || b * P != width || U->size(0) != b || U->size(2) != R || S->size(0) != b || S->size(1) != b || S->size(2) != R) return false;
    pr.U = U->data_ptr(), pr.V = V->data_ptr(), pr.S = S->data_ptr();
    if (PyTuple_GET_ITEM(o, 3) != Py_None) {
      const at::Tensor* t = d.factor(PyTuple_GET_ITEM(o, 3), d.dt);
      if (!t || t->numel() != b * Q || records_grad({t})) return false;
      pr.bias = t->data_ptr();
    }
    return true;
  }
  // (n, b Q) <- the rows at x
  void run(const Direct& d, const void* x, int64_t ldx, int act, const at::Tensor& out) {
    pr.out = out.data_ptr(), pr.ldo = b * Q;
    const Room w = d.ws(b, R);
    check_rc(blr_blast_multi(x, ldx, nullptr, BLR_ACT_NONE | act, d.n, d.code(), 1, &pr, b * R, R, 1, 16, 0, (int)b, (int)P, (int)Q, (int)R, w.ptr, w.bytes,
                             d.st));
  }
};

// attention(x, qkv, heads, weight, bias | None): self-attention of an encoder layer on x (B, T, d), more than 16 rows of it: qkv (Layer16, d -> 3 d) -> torch's
// scaled_dot_product_attention -> linear(weight, bias).
PyObject* py_attention(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  Direct d;
  Layer16 qkv;
  long heads;
  if (na != 5 || !d.take_x(a[0]) || d.x->dim() != 3 || d.n <= 16 || !take_ints(a + 2, 1, &heads) || heads < 1 || d.width % heads != 0) BLR_NONE();
  if (!qkv.take(d, a[1], d.width) || qkv.b * qkv.Q != 3 * d.width || records_grad({d.x})) BLR_NONE();
  const at::Tensor *W = plain(a[3]), *bias = a[4] == Py_None ? nullptr : plain(a[4]);
  if (!W || (a[4] != Py_None && !bias) || records_grad({W}) || (bias && records_grad({bias}))) BLR_NONE();
  const int64_t B = d.x->size(0), T = d.x->size(1), hd = d.width / heads, row = 3 * d.width;
  BLR_RECORD("attention", *d.x, *W);
  at::Tensor y;
  {
    NoGil free;
    const at::Tensor out = d.output(row);
    qkv.run(d, d.x->data_ptr(), d.ldx, 0, out);
    const int64_t size[4] = {B, heads, T, hd}, stride[4] = {T * row, hd, row, 1};
    const at::Tensor q = out.as_strided(size, stride, 0), k = out.as_strided(size, stride, d.width), v = out.as_strided(size, stride, 2 * d.width);
    const at::Tensor t = at::scaled_dot_product_attention(q, k, v).transpose(1, 2).reshape({B, T, d.width});
    y = bias ? at::linear(t, *W, *bias) : at::linear(t, *W);
  }
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// mlp(x, first, second, act): second(act(first(x))) of two Layer16, on more than 16 rows; act: BLR_ACT_OUT_*.
PyObject* py_mlp(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  Direct d;
  Layer16 first, second;
  long act;
  if (na != 4 || !d.take_x(a[0]) || d.n <= 16 || !take_ints(a + 3, 1, &act) || records_grad({d.x})) BLR_NONE();
  if (!first.take(d, a[1], d.width) || !second.take(d, a[2], first.b * first.Q)) BLR_NONE();
  BLR_RECORD("mlp", *d.x);
  at::Tensor out;
  {
    NoGil free;
    const at::Tensor mid = d.output(first.b * first.Q);
    first.run(d, d.x->data_ptr(), d.ldx, (int)act, mid);
    out = d.output(second.b * second.Q);
    second.run(d, mid.data_ptr(), first.b * first.Q, 0, out);
  }
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

PyMethodDef g_methods[] = {
    {"blast", (PyCFunction)(void*)py_blast, METH_FASTCALL, nullptr},
    {"blast_wq", (PyCFunction)(void*)py_blast_wq, METH_FASTCALL, nullptr},
    {"monarch", (PyCFunction)(void*)py_monarch, METH_FASTCALL, nullptr},
    {"low_rank", (PyCFunction)(void*)py_low_rank, METH_FASTCALL, nullptr},
    {"dense", (PyCFunction)(void*)py_dense, METH_FASTCALL, nullptr},
    {"multi", (PyCFunction)(void*)py_multi, METH_FASTCALL, nullptr},
    {"rmsnorm", (PyCFunction)(void*)py_rmsnorm, METH_FASTCALL, nullptr},
    {"layernorm", (PyCFunction)(void*)py_layernorm, METH_FASTCALL, nullptr},
    {"add_layernorm", (PyCFunction)(void*)py_add_layernorm, METH_FASTCALL, nullptr},
    {"attention", (PyCFunction)(void*)py_attention, METH_FASTCALL, nullptr},
    {"mlp", (PyCFunction)(void*)py_mlp, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_blr_torch", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__blr_torch(void) { return PyModule_Create(&g_module); }
