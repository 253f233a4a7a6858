// The single-GPU call of the public functions, host side in C++: one autograd function that allocates the
// results, fills the C ABI's parameter structs and launches.
//
// A training step on a few thousand tokens takes the GPU 40-300 us; through Python and ctypes (the ring's path,
// ring_swa/_ring.py) it took the host more -- the interpreter in the autograd engine's thread, a field-by-field
// ctypes struct, torch's Python tensor constructors -- and the GPU waited.  Host time of a call on 128 tokens: forward
// 10 us here and 47 there; a step through torch.autograd.grad 83 and 386, of which the engine and its
// thread take 51 (measured with an autograd function that does nothing, in the same loop).
//
// attention() returns None whenever a call is not an ordinary one (see `ordinary`: other dtypes or devices, a trace, a
// transform, a forward-mode tangent, an error to report, no status word yet) or its tensors are of another
// Python type: the Python path then runs it, or raises what it raises.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <cmath>
#include <cstring>

#include "../../include/rswa.h"

namespace {

constexpr int kMaxDevices = 64;
constexpr int64_t kHeadDim = 128, kNarrowHeadDim = 64;  // the widths that have kernels
// per device: the status word the kernels raise and its host mirror (made by new_status)
int32_t* g_status[kMaxDevices] = {nullptr};
const volatile int32_t* g_mirror[kMaxDevices] = {nullptr};

// [tokens, heads, D] (packed sequences) or [batch, tokens, heads, D]
struct Dims {
  int64_t batch, tokens, heads;
};
Dims dims_of(const at::Tensor& t) {
  if (t.dim() == 3) return {1, t.size(0), t.size(1)};
  return {t.size(0), t.size(1), t.size(2)};
}
struct Strides {
  int64_t b, t, h;
};
Strides strides_of(const at::Tensor& t) {
  if (t.dim() == 3) return {0, t.stride(0), t.stride(1)};
  return {t.stride(0), t.stride(1), t.stride(2)};
}

// The kernels address tensors through TMA descriptors: positive strides in multiples of 16 bytes, the head
// dimension contiguous.  Anything else (expanded gradients, odd slices) is copied.
bool dense_enough(const at::Tensor& t) {
  const auto st = t.strides();
  if (st.back() != 1 || (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) != 0) return false;
  for (size_t i = 0; i + 1 < st.size(); ++i)
    if (st[i] <= 0 || st[i] % 8 != 0) return false;
  return true;
}
at::Tensor dense(const at::Tensor& t) {
  if (dense_enough(t)) return t;
  const at::Tensor c = t.contiguous();
  // contiguous() returns a tensor that is contiguous already as it is, unaligned or with odd strides of its
  // dimensions of size 1.  The library refuses those at 128 elements per head; at 64 they are copied, as by the
  // zero padding that other widths go through.
  const bool batch_of_one = t.dim() == 4 && t.size(0) == 1 && t.stride(0) == 0;  // (the library knows what to do)
  if (t.size(-1) == kNarrowHeadDim && c.data_ptr() == t.data_ptr() && !dense_enough(batch_of_one ? c.select(0, 0) : c))
    return t.clone(at::MemoryFormat::Contiguous);
  return c;
}

struct Call {
  int64_t window, n_sink;
  double scale;
};

void fill_geom(rswa_geom_t& g, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& cu, const Call& c) {
  const Dims dq = dims_of(q), dk = dims_of(k);
  const Strides sk = strides_of(k);
  g.dtype = q.scalar_type() == at::kBFloat16 ? RSWA_DTYPE_BF16 : RSWA_DTYPE_FP16;
  g.batch = static_cast<int32_t>(dq.batch);
  g.q_len = static_cast<int32_t>(dq.tokens);
  g.n_q_heads = static_cast<int32_t>(dq.heads);
  g.n_kv_heads = static_cast<int32_t>(dk.heads);
  g.head_dim = static_cast<int32_t>(q.size(-1));
  g.window = static_cast<int32_t>(c.window);
  g.n_sink = static_cast<int32_t>(c.n_sink);
  g.softmax_scale = static_cast<float>(c.scale);
  if (cu.defined()) {
    g.cu_seqlens = cu.const_data_ptr<int32_t>();
    g.n_seqs = static_cast<int32_t>(cu.numel() - 1);
  }
  g.n_spans = 1;
  rswa_span_t& s = g.spans[0];
  s.k = k.data_ptr();
  s.v = v.data_ptr();
  s.kv_stride_b = sk.b, s.kv_stride_t = sk.t, s.kv_stride_h = sk.h;
  s.len = static_cast<int32_t>(dk.tokens);
}

void check(int rc, const char* what) {
  if (rc == RSWA_OK) return;
  if (rc == RSWA_E_ARG || rc == RSWA_E_UNSUPPORTED) TORCH_CHECK_VALUE(false, what, ": ", rswa_last_error());
  TORCH_CHECK(false, what, ": ", rswa_last_error(), " (code ", rc, ")");
}

// q, k, v (and cu_seqlens) are what the kernels take and fit together.
bool fits(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& cu) {
  if (!q.is_cuda() || q.layout() != at::kStrided || k.layout() != at::kStrided || v.layout() != at::kStrided) return false;
  if (q.scalar_type() != at::kBFloat16 && q.scalar_type() != at::kHalf) return false;
  if (k.scalar_type() != q.scalar_type() || v.scalar_type() != q.scalar_type()) return false;
  if (k.device() != q.device() || v.device() != q.device()) return false;
  if (q.dim() != (cu.defined() ? 3 : 4) || k.dim() != q.dim() || v.sizes() != k.sizes() || q.numel() == 0 || k.numel() == 0) return false;
  if ((q.size(-1) != kHeadDim && q.size(-1) != kNarrowHeadDim) || k.size(-1) != q.size(-1)) return false;
  const Dims dq = dims_of(q), dk = dims_of(k);
  if (dq.batch != dk.batch || dq.tokens != dk.tokens || dq.heads % dk.heads != 0) return false;
  if (dq.batch > 0x7fffffff || dq.tokens > 0x7fffffff || dq.heads > 0x7fffffff) return false;
  if (cu.defined() && (cu.device() != q.device() || cu.scalar_type() != at::kInt || cu.dim() != 1 || !cu.is_contiguous() || cu.numel() < 2))
    return false;
  return true;
}

bool ordinary(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& cu) {
  // A trace records what goes through the dispatcher: here the allocation of the output, not the kernels that fill
  // it.  The Python autograd function is recorded as one operator.
  if (torch::jit::tracer::isTracing()) return false;
  // vmap, torch.func.grad and the like: the Python autograd function says that it does not support them
  if (c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode)) return false;
  // forward-mode derivatives: there are none, and the Python autograd function says so
  for (const at::Tensor* t : {&q, &k, &v})
    if (t->_fw_grad(0).defined()) return false;
  if (!fits(q, k, v, cu)) return false;
  const int dev = q.get_device();
  if (dev < 0 || dev >= kMaxDevices || g_mirror[dev] == nullptr || *g_mirror[dev] != 0) return false;
  return dev == c10::cuda::current_device();
}

// Tensors that a saved-tensor hook hands back to the backward may be anything (another device, type, shape or
// layout than was saved): only those that the kernels can address are let through.
bool saved_as_expected(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& out, const at::Tensor& lse,
                       const at::Tensor& cu, const at::Tensor& dout) {
  if (!fits(q, k, v, cu) || q.sizes() != dout.sizes() || q.device() != dout.device() || q.scalar_type() != dout.scalar_type()) return false;
  if (out.sizes() != q.sizes() || out.scalar_type() != q.scalar_type() || out.device() != q.device()) return false;
  for (const at::Tensor* t : {&q, &k, &v, &out})
    if (t->stride(-1) != 1) return false;
  const Dims d = dims_of(q);
  return k.strides() == v.strides() && lse.sizes() == at::IntArrayRef({d.batch, d.heads, d.tokens}) && lse.scalar_type() == at::kFloat &&
         lse.device() == q.device() && lse.is_contiguous();
}

at::Tensor forward(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& cu, const Call& c, at::Tensor& lse) {
  const Dims d = dims_of(q);
  at::Tensor out = at::empty_like(q);
  lse = at::empty({d.batch, d.heads, d.tokens}, q.options().dtype(at::kFloat));
  rswa_fwd_params_t p;
  std::memset(&p, 0, sizeof(p));
  fill_geom(p.g, q, k, v, cu, c);
  const Strides sq = strides_of(q), so = strides_of(out);
  p.q = q.data_ptr();
  p.q_stride_b = sq.b, p.q_stride_t = sq.t, p.q_stride_h = sq.h;
  p.out = out.data_ptr();
  p.o_stride_b = so.b, p.o_stride_t = so.t, p.o_stride_h = so.h;
  p.lse = lse.data_ptr<float>();
  p.lse_stride_b = d.heads * d.tokens, p.lse_stride_h = d.tokens;
  p.status = g_status[q.get_device()];
  const auto call = q.size(-1) == kNarrowHeadDim ? rswa_fwd_d64 : rswa_fwd;
  check(call(&p, c10::cuda::getCurrentCUDAStream(q.get_device()).stream()), "rswa_fwd");
  return out;
}

class SwaFunction : public torch::autograd::Function<SwaFunction> {
 public:
  static at::Tensor forward(torch::autograd::AutogradContext* ctx, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v,
                            const std::optional<at::Tensor>& cu_, int64_t window, int64_t n_sink, double scale) {
    const at::Tensor cu = cu_.has_value() ? *cu_ : at::Tensor();
    at::Tensor lse;
    at::Tensor out = ::forward(q, k, v, cu, {window, n_sink, scale}, lse);
    ctx->save_for_backward({q, k, v, out, lse, cu});
    ctx->saved_data["window"] = window;
    ctx->saved_data["n_sink"] = n_sink;
    ctx->saved_data["scale"] = scale;
    return out;
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const at::Tensor &q = saved[0], &k = saved[1], &v = saved[2], &out = saved[3], &lse = saved[4], &cu = saved[5];
    const Call c = {ctx->saved_data["window"].toInt(), ctx->saved_data["n_sink"].toInt(), ctx->saved_data["scale"].toDouble()};
    TORCH_CHECK_VALUE(saved_as_expected(q, k, v, out, lse, cu, grads[0]),
                      "rswa_bwd: a saved tensor came back from a hook on another device or with another type, shape or layout");
    const c10::cuda::CUDAGuard guard(q.device());
    const at::Tensor dout = dense(grads[0]);
    at::Tensor dq = at::empty_like(q);
    at::Tensor dk = at::empty(k.sizes(), k.options()), dv = at::empty(k.sizes(), k.options());
    const Dims d = dims_of(q);
    const int64_t hkv = dims_of(k).heads;
    int64_t ws_bytes = rswa_bwd_workspace_bytes(d.batch, d.tokens, d.heads, kHeadDim);
    if (c.n_sink > 0) ws_bytes += rswa_bwd_sink_workspace_bytes(d.batch, d.tokens, hkv, c.window, c.n_sink, cu.defined() ? cu.numel() - 1 : 0);
    at::Tensor ws = at::empty({ws_bytes}, q.options().dtype(at::kByte));

    rswa_bwd_params_t p;
    std::memset(&p, 0, sizeof(p));
    fill_geom(p.g, q, k, v, cu, c);
    rswa_span_t& s = p.g.spans[0];
    const Strides skv = strides_of(dk);
    s.dk = dk.data_ptr();
    s.dv = dv.data_ptr();
    s.dkv_stride_b = skv.b, s.dkv_stride_t = skv.t, s.dkv_stride_h = skv.h;
    const Strides sq = strides_of(q), so = strides_of(out), sd = strides_of(dout), sdq = strides_of(dq);
    p.q = q.data_ptr();
    p.q_stride_b = sq.b, p.q_stride_t = sq.t, p.q_stride_h = sq.h;
    p.out = out.data_ptr();
    p.o_stride_b = so.b, p.o_stride_t = so.t, p.o_stride_h = so.h;
    p.dout = dout.data_ptr();
    p.do_stride_b = sd.b, p.do_stride_t = sd.t, p.do_stride_h = sd.h;
    p.lse = lse.data_ptr<float>();
    p.lse_stride_b = d.heads * d.tokens, p.lse_stride_h = d.tokens;
    p.dq = dq.data_ptr();
    p.dq_stride_b = sdq.b, p.dq_stride_t = sdq.t, p.dq_stride_h = sdq.h;
    p.workspace = ws.data_ptr();
    p.workspace_bytes = ws_bytes;
    p.flags = RSWA_BWD_INIT | RSWA_BWD_FINISH;
    p.status = g_status[q.get_device()];
    const auto call = q.size(-1) == kNarrowHeadDim ? rswa_bwd_d64 : rswa_bwd;
    check(call(&p, c10::cuda::getCurrentCUDAStream(q.get_device()).stream()), "rswa_bwd");
    return {dq, dk, dv, at::Tensor(), at::Tensor(), at::Tensor(), at::Tensor()};
  }
};

// attention(q, k, v, window, n_sink, scale or None, cu_seqlens or None) -> out, or None (see above)
PyObject* py_attention(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 7) {
    PyErr_SetString(PyExc_TypeError, "attention takes 7 arguments");
    return nullptr;
  }
  for (int i = 0; i < 3; ++i)  // (Tensor or Parameter: the result of another subclass is of that type)
    if (!THPVariable_CheckTypeExact(Py_TYPE(args[i]))) Py_RETURN_NONE;
  if (args[6] != Py_None && !THPVariable_Check(args[6])) Py_RETURN_NONE;
  const int64_t window = PyLong_AsLongLong(args[3]), n_sink = PyLong_AsLongLong(args[4]);
  double scale = args[5] == Py_None ? 0. : PyFloat_AsDouble(args[5]);
  if (PyErr_Occurred()) {  // numbers of other types: Python knows how to convert them, or what to raise
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  at::Tensor q = THPVariable_Unpack(args[0]), k = THPVariable_Unpack(args[1]), v = THPVariable_Unpack(args[2]);
  const at::Tensor cu = args[6] == Py_None ? at::Tensor() : THPVariable_Unpack(args[6]);
  if (window < 0 || window > 0x7fffffff || n_sink < 0 || n_sink > 0x7fffffff || !ordinary(q, k, v, cu)) Py_RETURN_NONE;
  if (args[5] == Py_None) scale = 1. / std::sqrt(static_cast<double>(q.size(-1)));
  at::Tensor out;
  {
    pybind11::gil_scoped_release no_gil;
    q = dense(q);
    k = dense(k);
    v = dense(v);
    if (k.strides() != v.strides()) {
      k = k.contiguous();
      v = v.contiguous();
      if (k.strides() != v.strides()) {  // (in dimensions of size 1)
        k = k.clone(at::MemoryFormat::Contiguous);
        v = v.clone(at::MemoryFormat::Contiguous);
      }
    }
    if (at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad())) {
      out = SwaFunction::apply(q, k, v, cu.defined() ? std::optional<at::Tensor>(cu) : std::nullopt, window, n_sink, scale);
    } else {
      at::Tensor lse;
      out = forward(q, k, v, cu, {window, n_sink, scale}, lse);
    }
  }
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// new_status(device index) -> (status word, its host mirror): two int32 tensors of one element that live as long as
// the process.  Not from torch's allocators: the first call on a device may be inside a stream capture, whose
// allocations belong to the graph (the word would be cleared by every replay) and which allows no pinned ones.
PyObject* py_new_status(PyObject*, PyObject* arg) {
  HANDLE_TH_ERRORS
  const long dev = PyLong_AsLong(arg);
  if (PyErr_Occurred()) return nullptr;
  TORCH_CHECK_VALUE(dev >= 0 && dev < kMaxDevices, "device index ", dev, " is outside the ", kMaxDevices, " this module has status words for");
  int32_t *word = nullptr, *mirror = nullptr;
  {
    const c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(dev));
    const c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);
    C10_CUDA_CHECK(cudaMalloc(&word, sizeof(int32_t)));
    C10_CUDA_CHECK(cudaHostAlloc(&mirror, sizeof(int32_t), cudaHostAllocPortable | cudaHostAllocMapped));
    *mirror = 0;
    cudaStream_t stream;  // (of its own: the current one may be capturing)
    C10_CUDA_CHECK(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
    C10_CUDA_CHECK(cudaMemsetAsync(word, 0, sizeof(int32_t), stream));
    C10_CUDA_CHECK(cudaStreamSynchronize(stream));
    C10_CUDA_CHECK(cudaStreamDestroy(stream));
  }
  check(rswa_set_status_mirror(word, mirror), "rswa_set_status_mirror");
  g_status[dev] = word;
  g_mirror[dev] = mirror;
  const auto options = at::TensorOptions().dtype(at::kInt);
  return Py_BuildValue("(NN)", THPVariable_Wrap(at::from_blob(word, {1}, options.device(at::kCUDA, static_cast<c10::DeviceIndex>(dev)))),
                       THPVariable_Wrap(at::from_blob(mirror, {1}, options)));
  END_HANDLE_TH_ERRORS
}

PyMethodDef g_methods[] = {
    {"attention", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_attention)), METH_FASTCALL,
     "attention(q, k, v, window, n_sink, scale, cu_seqlens) -> out or None (the call is not for this path)"},
    {"new_status", py_new_status, METH_O, "new_status(device_index) -> (status word, host mirror)"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_native", "Single-GPU host path of ring_swa", -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&g_module); }
