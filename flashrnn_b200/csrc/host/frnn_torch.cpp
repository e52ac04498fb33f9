// The Python front end's way into libfrnn_b200.so: argument checks, output allocation, the autograd node and the decoding
// step in native code.  A call of the Python version of this path (torch.autograd.Function, ctypes structures, one Python
// object per pointer) took 45 us of host time for an inference pass, 220 us for a training pass -- more than the kernels of a
// small problem -- and 10 us for a decoding step.
//
// The library's entry points are handed in as addresses (see `init`), so this module links against torch only and follows
// whichever build of the library the package loaded.  Everything unusual -- a wrong shape, an unknown name, other layouts,
// a process group -- is left to the Python code: `call` then returns None.
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>
#include <torch/torch.h>

#include <cstring>
#include <string>

#include "../../../include/frnn.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

struct Api {
  int (*query)(const frnn_problem*, frnn_plan*) = nullptr;
  int (*query_tile)(const frnn_problem*, int, int, int, frnn_plan*) = nullptr;
  int (*forward)(const frnn_plan*, const frnn_fwd_args*, void*) = nullptr;
  int (*backward)(const frnn_plan*, const frnn_bwd_args*, void*) = nullptr;
  int (*finalize)(const frnn_plan*, const void*, void*, void*, void*) = nullptr;
  const char* (*text)(int) = nullptr;
} api;

void check(const char* what, int code) {
  TORCH_CHECK(code == 0, what, " failed with status ", code, ": ", api.text(code));
}

// gate and state counts: flashrnn/flashrnn/flashrnn.py:49-71 of the reference
struct Cell { const char* name; int id; int64_t Gr, Gw, Gt, S; };
constexpr Cell kCells[] = {{"lstm", FRNN_CELL_LSTM, 4, 4, 4, 2}, {"gru", FRNN_CELL_GRU, 3, 3, 4, 1},
                           {"elman", FRNN_CELL_ELMAN, 1, 1, 1, 1}, {"slstm", FRNN_CELL_SLSTM, 4, 4, 4, 4}};
const Cell* find_cell(const char* name) {
  for (const Cell& c : kCells)
    if (!std::strcmp(c.name, name)) return &c;
  return nullptr;
}

at::ScalarType kernel_type(const char* name) {
  if (!std::strcmp(name, "bfloat16")) return at::kBFloat16;
  if (!std::strcmp(name, "float16")) return at::kHalf;
  if (!std::strcmp(name, "float32")) return at::kFloat;
  return at::ScalarType::Undefined;
}
int dtype_id(at::ScalarType t) { return t == at::kFloat ? FRNN_DTYPE_F32 : t == at::kHalf ? FRNN_DTYPE_F16 : FRNN_DTYPE_BF16; }

// What a call needs beside its tensors.
struct Call {
  int cell = 0;
  int64_t S = 0;
  at::ScalarType kdt = at::kBFloat16, sdt = at::kBFloat16;  // kernel and state element types
  double forward_clip = 0, grad_clip = 0;
  bool cut = false, training = false;
  int cluster_size = 0, batch_tile = 0;
};

// A 5-d tensor the kernels may read through strides (innermost dimension contiguous, the others non-negative multiples of 8
// elements, 16-byte aligned) as it is, anything else as a dense copy with all-zero strides.
Tensor kernel_view(const Tensor& t, at::ScalarType dt, int64_t (&stride)[4]) {
  std::memset(stride, 0, sizeof(stride));
  if (t.scalar_type() == dt && t.dim() == 5 && t.stride(4) == 1 && !t.is_contiguous() && reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0) {
    bool fits = true, any = false;
    for (int i = 0; i < 4; ++i) {
      fits = fits && t.stride(i) >= 0 && t.stride(i) % 8 == 0;
      any = any || t.stride(i) != 0;
    }
    if (fits && any) {
      for (int i = 0; i < 4; ++i) stride[i] = t.stride(i);
      return t;
    }
  }
  return t.to(dt).contiguous();
}

void* stream_of(const at::Device& d) { return c10::cuda::getCurrentCUDAStream(d.index()).stream(); }

struct Forward {
  frnn_plan plan;
  Tensor R, s0, states, cache, ws;
};

Forward run_forward(const Tensor& Wx, const Tensor& R, const Tensor& b, const Tensor& s0, const Call& c) {
  const int64_t B = Wx.size(0), T = Wx.size(1), N = Wx.size(3), D = Wx.size(4);
  Forward f = {};
  frnn_fwd_args a = {};
  const Tensor Wx_k = kernel_view(Wx, c.kdt, a.wx_stride), b_k = b.to(c.kdt).contiguous();
  f.R = R.to(c.kdt).contiguous();
  const c10::cuda::CUDAGuard guard(Wx.device());
  void* stream = stream_of(Wx.device());
  const auto opt = at::TensorOptions().device(Wx.device());
  f.s0 = s0.to(c.sdt).contiguous();
  frnn_problem pr = {};
  pr.cell = c.cell;
  pr.B = (int32_t)B; pr.T = (int32_t)T; pr.N = (int32_t)N; pr.D = (int32_t)D;
  pr.dtype_io = dtype_id(c.kdt);
  pr.dtype_state = dtype_id(c.sdt);
  pr.training = c.training;
  pr.forward_clip = (float)c.forward_clip;
  pr.grad_clip = (float)c.grad_clip;
  pr.grad_cut = c.cut;
  if (c.cluster_size || c.batch_tile) check("frnn_query_tile", api.query_tile(&pr, c.cluster_size, c.batch_tile, 0, &f.plan));
  else check("frnn_query", api.query(&pr, &f.plan));
  f.states = at::empty({c.S, B, T, N, D}, opt.dtype(c.sdt));
  if (c.training) f.cache = at::empty({(int64_t)std::max<uint64_t>(f.plan.cache_bytes, 16)}, opt.dtype(at::kByte));
  f.ws = at::empty({(int64_t)f.plan.workspace_bytes}, opt.dtype(at::kByte));
  a.Wx = Wx_k.const_data_ptr(); a.R = f.R.const_data_ptr(); a.b = b_k.const_data_ptr(); a.s0 = f.s0.const_data_ptr();
  a.states = f.states.data_ptr();
  a.cache = c.training ? f.cache.data_ptr() : nullptr;
  a.workspace = f.ws.data_ptr();
  check("frnn_forward", api.forward(&f.plan, &a, stream));
  return f;
}

// One frnn_forward, one frnn_backward + frnn_finalize_grads: the place of FlashRNNFunctionFused (reference
// flashrnn.py:688-801).  No torch operator that autocast could re-type runs inside.
struct FrnnNode : public torch::autograd::Function<FrnnNode> {
  struct Kept {  // what the reverse pass needs to know of the forward call
    frnn_plan plan;
    int64_t Gw, Gt;
    at::ScalarType types[4];  // of the inputs: the gradients' types
  };
  static Tensor forward(AutogradContext* ctx, const Tensor& Wx, const Tensor& R, const Tensor& b, const Tensor& s0, const Call& c) {
    Forward f = run_forward(Wx, R, b, s0, c);
    ctx->save_for_backward({f.R, f.s0, f.states, f.cache, f.ws});
    Kept k{f.plan, Wx.size(2), b.size(0), {Wx.scalar_type(), R.scalar_type(), b.scalar_type(), s0.scalar_type()}};
    ctx->saved_data["call"] = std::string(reinterpret_cast<const char*>(&k), sizeof(k));
    return f.states;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &R = saved[0], &s0 = saved[1], &states = saved[2], &cache = saved[3], &ws = saved[4];
    Kept k;
    std::memcpy(&k, ctx->saved_data["call"].toStringRef().data(), sizeof(k));
    const frnn_plan& plan = k.plan;
    const c10::cuda::CUDAGuard guard(states.device());
    void* stream = stream_of(states.device());
    frnn_bwd_args a = {};
    const Tensor ds = grads[0].defined() ? kernel_view(grads[0], states.scalar_type(), a.dstates_stride) : at::zeros_like(states);
    const int64_t N = plan.prob.N, D = plan.prob.D;
    const auto opt = R.options().requires_grad(false);
    Tensor dWx = at::empty({plan.prob.B, plan.prob.T, k.Gw, N, D}, opt);
    Tensor ds0 = at::empty(s0.sizes(), s0.options().requires_grad(false)), dR = at::empty(R.sizes(), opt);
    Tensor db = at::empty({k.Gt, N, D}, opt);
    a.R = R.const_data_ptr(); a.s0 = s0.const_data_ptr(); a.states = states.const_data_ptr();
    a.cache = cache.const_data_ptr(); a.dstates = ds.const_data_ptr();
    a.dWx = dWx.data_ptr(); a.ds0 = ds0.data_ptr();
    a.workspace = ws.data_ptr();
    check("frnn_backward", api.backward(&plan, &a, stream));
    check("frnn_finalize_grads",
          api.finalize(&plan, static_cast<const char*>(ws.const_data_ptr()) + plan.grads_offset, dR.data_ptr(), db.data_ptr(), stream));
    return {dWx.to(k.types[0]), dR.to(k.types[1]), db.to(k.types[2]), ds0.to(k.types[3]), Tensor()};
  }
};

// -> (states, last), or an undefined pair where the Python code has to look at the call
std::pair<Tensor, Tensor> run_call(const Tensor& Wx, const Tensor& R, const Tensor& b, Tensor s0, Call& c) {
  if (!s0.defined()) {
    const c10::cuda::CUDAGuard guard(Wx.device());
    s0 = at::empty({c.S, Wx.size(0), 1, Wx.size(3), Wx.size(4)}, at::TensorOptions().device(Wx.device()).dtype(c.sdt));
    TORCH_CHECK(cudaMemsetAsync(s0.data_ptr(), 0, s0.nbytes(), static_cast<cudaStream_t>(stream_of(Wx.device()))) == cudaSuccess,
                "flashrnn_b200: cudaMemsetAsync failed");
  }
  c.training = at::GradMode::is_enabled() && (Wx.requires_grad() || R.requires_grad() || b.requires_grad() || s0.requires_grad());
  Tensor states;
  if (c.training) {
    states = FrnnNode::apply(Wx, R, b, s0, c);
  } else {
    const at::NoGradGuard no_grad;
    states = run_forward(Wx, R, b, s0, c).states;
  }
  return {states, states.narrow(2, states.size(2) - 1, 1)};
}

bool is(const Tensor& t, std::initializer_list<int64_t> shape) { return t.sizes().equals(at::IntArrayRef(shape.begin(), shape.size())); }

Tensor tensor_arg(PyObject* o) { return THPVariable_Check(o) ? THPVariable_Unpack(o) : Tensor(); }

PyObject* pack(const std::pair<Tensor, Tensor>& r) {
  THPObjectPtr t(PyTuple_New(2));
  if (!t) throw python_error();
  PyTuple_SET_ITEM(t.get(), 0, THPVariable_Wrap(r.first));
  PyTuple_SET_ITEM(t.get(), 1, THPVariable_Wrap(r.second));
  return t.release();
}

// call(Wx, R, b, states or None, function, dtype): flashrnn() with default configuration and layouts.  None where a check fails.
PyObject* py_call(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 6 || !PyUnicode_Check(args[4]) || !PyUnicode_Check(args[5])) Py_RETURN_NONE;
  const Tensor Wx = tensor_arg(args[0]), R = tensor_arg(args[1]), b = tensor_arg(args[2]), s0 = tensor_arg(args[3]);
  const Cell* cell = find_cell(PyUnicode_AsUTF8(args[4]));
  Call c;
  c.kdt = kernel_type(PyUnicode_AsUTF8(args[5]));
  if (!api.forward || !cell || c.kdt == at::ScalarType::Undefined || !Wx.defined() || !R.defined() || !b.defined() ||
      (!s0.defined() && args[3] != Py_None))
    Py_RETURN_NONE;
  if (!Wx.is_cuda() || R.device() != Wx.device() || b.device() != Wx.device() || (s0.defined() && s0.device() != Wx.device()) || Wx.dim() != 5)
    Py_RETURN_NONE;
  const int64_t B = Wx.size(0), T = Wx.size(1), N = Wx.size(3), D = Wx.size(4);
  if (T == 0 || Wx.size(2) != cell->Gw || !is(R, {cell->Gr, N, D, D}) || !is(b, {cell->Gt, N, D}) || (s0.defined() && !is(s0, {cell->S, B, 1, N, D})))
    Py_RETURN_NONE;
  auto known = [](at::ScalarType t) { return t == at::kBFloat16 || t == at::kHalf || t == at::kFloat; };
  if (!known(Wx.scalar_type()) || !known(R.scalar_type()) || !known(b.scalar_type())) Py_RETURN_NONE;
  // states live in the kernel type, or in float32 when Wx or the given states do
  const bool f32 = c.kdt == at::kFloat || Wx.scalar_type() == at::kFloat || (s0.defined() && s0.scalar_type() == at::kFloat);
  c.sdt = f32 ? at::kFloat : c.kdt;
  c.cell = cell->id;
  c.S = cell->S;
  std::pair<Tensor, Tensor> r;
  {
    pybind11::gil_scoped_release nogil;
    r = run_call(Wx, R, b, s0, c);
  }
  return pack(r);
  END_HANDLE_TH_ERRORS
}

// run(Wx, R, b, states, function, dtype, dtype_s, forward_clip, grad_clip, cut, cluster_size, batch_tile): checked arguments in
// the native layouts
PyObject* py_run(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 12 && api.forward, "flashrnn_b200: bad native call");
  const Tensor Wx = tensor_arg(args[0]), R = tensor_arg(args[1]), b = tensor_arg(args[2]), s0 = tensor_arg(args[3]);
  TORCH_CHECK(Wx.defined() && R.defined() && b.defined() && (s0.defined() || args[3] == Py_None), "flashrnn_b200: expected tensors");
  const Cell* cell = find_cell(PyUnicode_AsUTF8(args[4]));
  Call c;
  c.kdt = kernel_type(PyUnicode_AsUTF8(args[5]));
  c.sdt = kernel_type(PyUnicode_AsUTF8(args[6]));
  TORCH_CHECK(cell && c.kdt != at::ScalarType::Undefined && c.sdt != at::ScalarType::Undefined, "flashrnn_b200: unknown function or dtype");
  c.cell = cell->id;
  c.S = cell->S;
  c.forward_clip = PyFloat_AsDouble(args[7]);
  c.grad_clip = PyFloat_AsDouble(args[8]);
  c.cut = PyObject_IsTrue(args[9]) == 1;
  c.cluster_size = (int)PyLong_AsLong(args[10]);
  c.batch_tile = (int)PyLong_AsLong(args[11]);
  if (PyErr_Occurred()) throw python_error();
  std::pair<Tensor, Tensor> r;
  {
    pybind11::gil_scoped_release nogil;
    r = run_call(Wx, R, b, s0, c);
  }
  return pack(r);
  END_HANDLE_TH_ERRORS
}

// ---- decoding: one handle per FlashRNNStepper
struct Stepper {
  frnn_plan plan;
  frnn_fwd_args args;
  Tensor R, b, s0, out, ws;
  at::ScalarType kdt;
  int64_t shape[5];
};
constexpr const char* kStepperName = "flashrnn_b200.stepper";

// stepper(R, b, s0, out, ws, plan bytes, (B, chunk, Gw, N, D)) -> handle
PyObject* py_stepper(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 7 && api.forward && PyBytes_Check(args[5]) && PyBytes_GET_SIZE(args[5]) == (Py_ssize_t)sizeof(frnn_plan), "flashrnn_b200: bad native call");
  auto s = std::make_unique<Stepper>();
  s->R = tensor_arg(args[0]); s->b = tensor_arg(args[1]); s->s0 = tensor_arg(args[2]); s->out = tensor_arg(args[3]); s->ws = tensor_arg(args[4]);
  std::memcpy(&s->plan, PyBytes_AS_STRING(args[5]), sizeof(frnn_plan));
  for (int i = 0; i < 5; ++i) s->shape[i] = PyLong_AsLongLong(PyTuple_GetItem(args[6], i));
  if (PyErr_Occurred()) throw python_error();
  s->kdt = s->R.scalar_type();
  s->args = {};
  s->args.R = s->R.const_data_ptr(); s->args.b = s->b.const_data_ptr(); s->args.s0 = s->s0.data_ptr();
  s->args.states = s->out.data_ptr(); s->args.workspace = s->ws.data_ptr();
  s->args.last = s->s0.data_ptr();  // the carried states are updated in place by the library call
  return PyCapsule_New(s.release(), kStepperName, [](PyObject* c) { delete static_cast<Stepper*>(PyCapsule_GetPointer(c, kStepperName)); });
  END_HANDLE_TH_ERRORS
}

// step(handle, Wx) -> True, or False where Wx is not what the stepper takes
PyObject* py_step(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 2, "flashrnn_b200: bad native call");
  Stepper* s = static_cast<Stepper*>(PyCapsule_GetPointer(args[0], kStepperName));
  if (!s) throw python_error();
  const Tensor Wx = tensor_arg(args[1]);
  if (!Wx.defined() || Wx.scalar_type() != s->kdt || Wx.device() != s->R.device() || !Wx.sizes().equals(at::IntArrayRef(s->shape, 5)) || !Wx.is_contiguous())
    Py_RETURN_FALSE;
  frnn_fwd_args a = s->args;
  a.Wx = Wx.const_data_ptr();
  {
    pybind11::gil_scoped_release nogil;
    const c10::cuda::CUDAGuard guard(Wx.device());
    check("frnn_forward", api.forward(&s->plan, &a, stream_of(Wx.device())));
  }
  s->plan.keep_packed_r = 1;
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

// init(addresses of frnn_query, frnn_query_tile, frnn_forward, frnn_backward, frnn_finalize_grads, frnn_status_string)
PyObject* py_init(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 6, "flashrnn_b200: bad native call");
  void* p[6];
  for (int i = 0; i < 6; ++i) p[i] = PyLong_AsVoidPtr(args[i]);
  if (PyErr_Occurred()) throw python_error();
  api.query = reinterpret_cast<decltype(api.query)>(p[0]);
  api.query_tile = reinterpret_cast<decltype(api.query_tile)>(p[1]);
  api.backward = reinterpret_cast<decltype(api.backward)>(p[3]);
  api.finalize = reinterpret_cast<decltype(api.finalize)>(p[4]);
  api.text = reinterpret_cast<decltype(api.text)>(p[5]);
  api.forward = reinterpret_cast<decltype(api.forward)>(p[2]);
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

PyCFunction fast(PyObject* (*f)(PyObject*, PyObject* const*, Py_ssize_t)) { return reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(f)); }
PyMethodDef kMethods[] = {{"init", fast(py_init), METH_FASTCALL, nullptr},       {"call", fast(py_call), METH_FASTCALL, nullptr},
                          {"run", fast(py_run), METH_FASTCALL, nullptr},         {"stepper", fast(py_stepper), METH_FASTCALL, nullptr},
                          {"step", fast(py_step), METH_FASTCALL, nullptr},       {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_torch_bridge", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__torch_bridge(void) { return PyModule_Create(&kModule); }
