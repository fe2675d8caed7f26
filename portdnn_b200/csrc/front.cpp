// Native half of portdnn_b200/api.py: one function per operator that checks the tensors, allocates the
// result where the caller gave none and calls the C ABI on torch's current stream.  The checks are a
// handful of field reads in here; as Python they took 6-10 us per call, two to three times what the
// launch itself costs the host (api.conv2d 14.0 us against 4.0 us inside the library), and a network of
// short layers is bound by that: its host issues 55 calls before the device has run the first few.
//
// Every function takes exactly the arguments of the api.py function it stands behind, by position and
// in that order; names, defaults and documentation live there.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/portdnn_b200.h"

namespace {

// Thrown after a Python exception has been set.
struct PyFailure {};

[[noreturn]] void raise(PyObject* type, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  PyErr_FormatV(type, fmt, ap);
  va_end(ap);
  throw PyFailure();
}

// Runs f without the interpreter lock, as torch allocates and ctypes calls: a launch waits when the launch queue
// is full, an allocation when memory has to be found, and neither may keep the process's other threads from
// running (they may be what the queue waits for).  Costs the call 0.1 us.
template <typename F>
auto unlocked(F&& f) {
  struct Release {
    PyThreadState* state = PyEval_SaveThread();
    ~Release() { PyEval_RestoreThread(state); }
  } release;
  return f();
}

// A tensor argument; undefined for None.  (By value: the lock is released while it is in use.)
at::Tensor tensor(PyObject* o) {
  if (o == Py_None) return at::Tensor();
  if (!THPVariable_Check(o)) raise(PyExc_TypeError, "expected a torch.Tensor, got %.100s", Py_TYPE(o)->tp_name);
  return THPVariable_Unpack(o);
}

template <typename... T>
void require_cuda(const T&... ts) {
  const bool ok = ((!ts.defined() || (ts.is_cuda() && ts.is_contiguous())) && ...);
  if (!ok) raise(PyExc_ValueError, "tensors must be contiguous CUDA tensors");
}

int dtype_code(const at::Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return PDNN_F32;
    case at::kHalf: return PDNN_F16;
    case at::kBFloat16: return PDNN_BF16;
    default: raise(PyExc_KeyError, "unsupported dtype %s", c10::toString(t.scalar_type()));
  }
}

// A whole number.  (A text or a fraction is a mistake in the call: neither is turned into one.)
long integer(PyObject* o) {
  const long v = PyLong_AsLong(o);
  if (v == -1 && PyErr_Occurred()) throw PyFailure();
  return v;
}
// Whatever int() takes.
long to_integer(PyObject* o) {
  if (PyLong_CheckExact(o)) return integer(o);
  PyObject* n = PyNumber_Long(o);
  if (n == nullptr) throw PyFailure();
  const long v = PyLong_AsLong(n);
  Py_DECREF(n);
  if (v == -1 && PyErr_Occurred()) throw PyFailure();
  return v;
}
double real(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw PyFailure();
  return v;
}
bool truth(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw PyFailure();
  return v != 0;
}

// The bytes of a ctypes parameter structure.
template <typename P>
P params(PyObject* o) {
  Py_buffer view;
  if (PyObject_GetBuffer(o, &view, PyBUF_SIMPLE) != 0) throw PyFailure();
  P p;
  const bool fits = (size_t)view.len == sizeof(P);
  if (fits) memcpy(&p, view.buf, sizeof(P));
  PyBuffer_Release(&view);
  if (!fits) raise(PyExc_TypeError, "wrong parameter structure: %.100s", Py_TYPE(o)->tp_name);
  return p;
}

void* ptr(const at::Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// Calls the library, and reports its status as portdnn_b200.api does.  (The error text is the thread's own.)
template <typename F>
void call(F&& f) {
  const int status = unlocked(f);
  if (status == PDNN_OK) return;
  PyObject* api = PyImport_ImportModule("portdnn_b200.api");
  if (api != nullptr) {
    PyObject* r = PyObject_CallMethod(api, "_check", "i", status);
    Py_XDECREF(r);
    Py_DECREF(api);
  }
  if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, pdnn_last_error());
  throw PyFailure();
}

at::Tensor flat(int64_t n, const at::TensorOptions& options) { return unlocked([&] { return at::empty({n}, options); }); }
at::Tensor like(const at::Tensor& t) { return unlocked([&] { return at::empty_like(t); }); }

// `out` if the caller gave one, else a tensor of the shape of `like`.
at::Tensor out_or_like(const at::Tensor& out, const at::Tensor& t) { return out.defined() ? out : like(t); }

PyObject* conv2d(PyObject* const* a) {
  const long pass = integer(a[0]);
  const at::Tensor &inp = tensor(a[1]), &fil = tensor(a[2]);
  const PdnnConv2DParams p = params<PdnnConv2DParams>(a[3]);
  const int algorithm = (int)integer(a[4]);
  at::Tensor out = tensor(a[5]);
  const at::Tensor &workspace = tensor(a[6]), &bias = tensor(a[7]);
  const int activation = (int)integer(a[8]);
  const double alpha = real(a[9]), beta = real(a[10]);
  const at::Tensor& relu_out = tensor(a[11]);
  const bool output_f32 = truth(a[12]);
  const bool accumulate = truth(a[13]);
  const at::Tensor& bits = tensor(a[14]);
  const bool constant_filter = truth(a[15]), any_order = truth(a[16]);

  require_cuda(inp, fil, out, workspace, bias);
  const int64_t x = (int64_t)p.batch * p.in_rows * p.in_cols * p.channels;
  const int64_t w = (int64_t)p.window_rows * p.window_cols * (p.channels / (p.groups > 1 ? p.groups : 1)) * p.features;
  const int64_t y = (int64_t)p.batch * p.out_rows * p.out_cols * p.features;
  if (pass < 0 || pass > 2) raise(PyExc_KeyError, "%ld", pass);
  const int64_t n_in = pass == PDNN_INPUT_BACKPROP ? y : x, n_fil = pass == PDNN_FILTER_BACKPROP ? y : w;
  const int64_t n_out = pass == PDNN_FORWARD ? y : pass == PDNN_INPUT_BACKPROP ? x : w;
  if (inp.numel() != n_in || fil.numel() != n_fil)
    raise(PyExc_ValueError, "tensor sizes do not match the parameters: %lld/%lld, %lld/%lld", (long long)inp.numel(),
          (long long)n_in, (long long)fil.numel(), (long long)n_fil);
  require_cuda(bits);
  if (bits.defined()) {
    if (pass == PDNN_FILTER_BACKPROP)
      raise(PyExc_ValueError, "relu_bitmask belongs to the forward pass (output) and the input backprop (input)");
    if (bits.scalar_type() != at::kByte || bits.numel() * 8 != n_out)
      raise(PyExc_ValueError, "relu_bitmask must be a uint8 tensor of one bit per element");
  }
  const bool backprop_fused = relu_out.defined() || output_f32 || accumulate || (bits.defined() && pass != PDNN_FORWARD) ||
                              (constant_filter && pass == PDNN_INPUT_BACKPROP);
  if (backprop_fused && (pass == PDNN_FORWARD || (relu_out.defined() && pass != PDNN_INPUT_BACKPROP) ||
                         (output_f32 && pass != PDNN_FILTER_BACKPROP)))
    raise(PyExc_ValueError, "relu_forward_output belongs to the input backprop, output_f32 to the filter backprop");
  if (accumulate && !out.defined()) raise(PyExc_ValueError, "accumulate needs the tensor to add to as out");
  require_cuda(relu_out);
  const at::ScalarType out_type = output_f32 ? at::kFloat : inp.scalar_type();
  if (!out.defined()) out = flat(n_out, inp.options().dtype(out_type));
  if (out.numel() != n_out || out.scalar_type() != out_type)
    raise(PyExc_ValueError, "output tensor does not match the parameters");
  const size_t ws_elems = workspace.defined() ? (size_t)(workspace.nbytes() / inp.element_size()) : 0;
  const int dtype = dtype_code(inp);
  if (backprop_fused) {
    if (relu_out.defined() && relu_out.numel() != n_out)
      raise(PyExc_ValueError, "relu_forward_output must have the shape of the input gradient");
    PdnnBackpropFusion f = {};
    f.relu_forward_output = ptr(relu_out);
    f.output_f32 = output_f32;
    f.accumulate = (int)to_integer(a[13]);  // False / True, or 2 (dx already carries the mask)
    f.relu_bitmask = ptr(bits);
    f.constant_filter = constant_filter;
    call([&] {
      return pdnn_conv2d_backprop_fused((int)pass, dtype, ptr(inp), ptr(fil), ptr(out), &p, algorithm, &f, ptr(workspace),
                                        ws_elems, stream());
    });
    return THPVariable_Wrap(out);
  }
  const bool fused = bias.defined() || activation != PDNN_ACT_NONE || alpha != 1.0 || beta != 0.0 || bits.defined() ||
                     (constant_filter && pass == PDNN_FORWARD) || any_order;
  if (fused) {
    if (pass != PDNN_FORWARD) raise(PyExc_ValueError, "the fused epilogue exists for the forward pass only");
    PdnnConvEpilogue e = {};
    e.bias = ptr(bias);
    e.activation = activation;
    e.alpha = (float)alpha;
    e.beta = (float)beta;
    e.relu_bitmask = ptr(bits);
    e.constant_filter = constant_filter;
    e.any_order = any_order;
    call([&] {
      return pdnn_conv2d_fused(dtype, ptr(inp), ptr(fil), ptr(out), &p, algorithm, &e, ptr(workspace), ws_elems, stream());
    });
  } else {
    call([&] {
      return pdnn_conv2d((int)pass, dtype, ptr(inp), ptr(fil), ptr(out), &p, algorithm, ptr(workspace), ws_elems, stream());
    });
  }
  return THPVariable_Wrap(out);
}

PyObject* depthwise_conv2d(PyObject* const* a) {
  const long pass = integer(a[0]);
  const at::Tensor &inp = tensor(a[1]), &fil = tensor(a[2]);
  const PdnnDepthwiseConv2DParams p = params<PdnnDepthwiseConv2DParams>(a[3]);
  at::Tensor out = tensor(a[4]);
  const at::Tensor& workspace = tensor(a[5]);
  require_cuda(inp, fil, out, workspace);
  const int64_t x = (int64_t)p.batch * p.in_rows * p.in_cols * p.channels;
  const int64_t w = (int64_t)p.window_rows * p.window_cols * p.channels * p.channel_multiplier;
  const int64_t y = (int64_t)p.batch * p.out_rows * p.out_cols * p.channels * p.channel_multiplier;
  if (pass < 0 || pass > 2) raise(PyExc_KeyError, "%ld", pass);
  const int64_t n_in = pass == PDNN_INPUT_BACKPROP ? y : x, n_fil = pass == PDNN_FILTER_BACKPROP ? y : w;
  const int64_t n_out = pass == PDNN_FORWARD ? y : pass == PDNN_INPUT_BACKPROP ? x : w;
  if (inp.numel() != n_in || fil.numel() != n_fil) raise(PyExc_ValueError, "tensor sizes do not match the parameters");
  if (!out.defined()) out = flat(n_out, inp.options());
  const int dtype = dtype_code(inp);
  call([&] {
    return pdnn_depthwise_conv2d((int)pass, dtype, ptr(inp), ptr(fil), ptr(out), &p, ptr(workspace),
                                 workspace.defined() ? workspace.nbytes() : 0, stream());
  });
  return THPVariable_Wrap(out);
}

PyObject* pooling(PyObject* const* a) {
  const int op = (int)integer(a[0]), direction = (int)integer(a[1]);
  const at::Tensor& inp = tensor(a[2]);
  const PdnnPoolingParams p = params<PdnnPoolingParams>(a[3]);
  at::Tensor out = tensor(a[4]);
  require_cuda(inp, out);
  if (!out.defined()) {
    const int64_t px = direction == 0 ? (int64_t)p.out_rows * p.out_cols : (int64_t)p.in_rows * p.in_cols;
    out = flat(p.batch * px * p.channels, inp.options());
  }
  const int dtype = dtype_code(inp);
  call([&] { return pdnn_pooling(op, direction, dtype, ptr(inp), ptr(out), &p, stream()); });
  return THPVariable_Wrap(out);
}

PyObject* pooling_max_grad(PyObject* const* a) {
  const int op = (int)integer(a[0]);
  const at::Tensor &x = tensor(a[1]), &y = tensor(a[2]), &dy = tensor(a[3]);
  const PdnnPoolingParams p = params<PdnnPoolingParams>(a[4]);
  at::Tensor out = tensor(a[5]);
  const bool relu_input = truth(a[6]);
  require_cuda(x, y, dy, out);
  if (!out.defined()) out = flat(x.numel(), x.options());
  const int dtype = dtype_code(x);
  call([&] {
    return (relu_input ? pdnn_pooling_max_grad_relu : pdnn_pooling_max_grad)(op, dtype, ptr(x), ptr(y), ptr(dy), ptr(out), &p,
                                                                             stream());
  });
  return THPVariable_Wrap(out);
}

PyObject* pointwise(PyObject* const* a) {
  const int op = (int)integer(a[0]);
  const at::Tensor& inp = tensor(a[1]);
  require_cuda(inp, tensor(a[2]));
  const at::Tensor out = out_or_like(tensor(a[2]), inp);
  const int dtype = dtype_code(inp);
  call([&] { return pdnn_pointwise(op, dtype, ptr(inp), ptr(out), (size_t)inp.numel(), stream()); });
  return THPVariable_Wrap(out);
}

PyObject* pointwise_grad(PyObject* const* a) {
  const int op = (int)integer(a[0]);
  const at::Tensor &fwd = tensor(a[1]), &err = tensor(a[2]);
  require_cuda(fwd, err, tensor(a[3]));
  const at::Tensor out = out_or_like(tensor(a[3]), fwd);
  const int dtype = dtype_code(fwd);
  call([&] { return pdnn_pointwise_grad(op, dtype, ptr(fwd), ptr(err), ptr(out), (size_t)fwd.numel(), stream()); });
  return THPVariable_Wrap(out);
}

PyObject* bias_add(PyObject* const* a) {
  const at::Tensor &inp = tensor(a[0]), &bias = tensor(a[1]);
  const long channels = integer(a[2]);
  require_cuda(inp, bias, tensor(a[4]));
  if (channels == 0) raise(PyExc_ZeroDivisionError, "integer division or modulo by zero");
  const at::Tensor out = out_or_like(tensor(a[4]), inp);
  const int dtype = dtype_code(inp), activation = (int)to_integer(a[3]);
  call([&] {
    return pdnn_bias_add(dtype, ptr(inp), ptr(bias), ptr(out), (size_t)(inp.numel() / channels), (int)channels, activation,
                         stream());
  });
  return THPVariable_Wrap(out);
}

PyObject* scale_blend(PyObject* const* a) {
  const at::Tensor &x = tensor(a[0]), &b = tensor(a[2]);
  require_cuda(x, b, tensor(a[4]));
  const at::Tensor out = out_or_like(tensor(a[4]), x);
  const int dtype = dtype_code(x);
  const float alpha = (float)real(a[1]), beta = (float)real(a[3]);
  call([&] { return pdnn_scale_blend(dtype, ptr(x), alpha, ptr(b), beta, ptr(out), (size_t)x.numel(), stream()); });
  return THPVariable_Wrap(out);
}

// A sequence of extents: all are counted, the first kMostDims kept (the library takes no more than four).
constexpr int kMostDims = 16;
int extents(PyObject* o, int (&d)[kMostDims]) {
  PyObject* seq = PySequence_Fast(o, "expected a sequence of extents");
  if (seq == nullptr) throw PyFailure();
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(seq);
  for (Py_ssize_t i = 0; i < n && !PyErr_Occurred(); ++i) {
    PyObject* v = PyNumber_Long(PySequence_Fast_GET_ITEM(seq, i));
    const int extent = v != nullptr ? (int)PyLong_AsLong(v) : 0;
    Py_XDECREF(v);
    if (i < kMostDims) d[i] = extent;
  }
  Py_DECREF(seq);
  if (PyErr_Occurred()) throw PyFailure();
  return (int)n;
}

PyObject* binaryop(PyObject* const* a) {
  const int op = (int)to_integer(a[0]);
  const at::Tensor &lhs = tensor(a[1]), &rhs = tensor(a[3]);
  int ld[kMostDims] = {}, rd[kMostDims] = {};
  require_cuda(lhs, rhs, tensor(a[5]));
  const int nl = extents(a[2], ld), nr = extents(a[4], rd);
  at::Tensor out = tensor(a[5]);
  if (!out.defined()) {
    const int n = nl > nr ? nl : nr;
    int64_t numel = n <= kMostDims ? 1 : 0;  // (more than the library takes)
    for (int i = 0; i < n && numel != 0; ++i) {
      const int l = i < n - nl ? 1 : ld[i - (n - nl)], r = i < n - nr ? 1 : rd[i - (n - nr)];
      const int m = l > r ? l : r;
      numel *= m > 0 ? m : 0;
    }
    out = flat(numel, lhs.options());
  }
  const int dtype = dtype_code(lhs);
  call([&] { return pdnn_binaryop(op, dtype, ptr(lhs), ld, nl, ptr(rhs), rd, nr, ptr(out), stream()); });
  return THPVariable_Wrap(out);
}

PyObject* matmul(PyObject* const* a) {
  const at::Tensor &lhs = tensor(a[0]), &rhs = tensor(a[1]);
  auto extent = [](PyObject* o) {  // 8.0 is one, 8.5 is not
    return PyFloat_Check(o) && PyFloat_AS_DOUBLE(o) == (double)(int)PyFloat_AS_DOUBLE(o) ? to_integer(o) : integer(o);
  };
  const long batches = extent(a[2]), m = extent(a[3]), k = extent(a[4]), n = extent(a[5]);
  const bool tl = truth(a[6]), tr = truth(a[7]);
  const double beta = real(a[8]);
  at::Tensor out = tensor(a[9]);
  require_cuda(lhs, rhs, out);
  if (lhs.numel() != (int64_t)batches * m * k || rhs.numel() != (int64_t)batches * k * n)
    raise(PyExc_ValueError, "tensor sizes do not match the parameters");
  if (!out.defined()) {
    if (beta != 0.0) raise(PyExc_ValueError, "beta != 0 needs an output tensor to accumulate into");
    out = flat((int64_t)batches * m * n, lhs.options());
  }
  const int dtype = dtype_code(lhs);
  call([&] {
    return pdnn_matmul(dtype, tl, tr, ptr(lhs), ptr(rhs), ptr(out), (int)batches, (int)m, (int)k, (int)n, (float)beta, stream());
  });
  return THPVariable_Wrap(out);
}

PyObject* softmax(PyObject* const* a) {
  const at::Tensor &inp = tensor(a[0]), &gradient = tensor(a[5]);
  const long batch = integer(a[1]), rows = integer(a[2]), cols = integer(a[3]), channels = integer(a[4]);
  require_cuda(inp, gradient, tensor(a[6]));
  if (inp.numel() != (int64_t)batch * rows * cols * channels)
    raise(PyExc_ValueError, "tensor size does not match the parameters");
  const at::Tensor out = out_or_like(tensor(a[6]), inp);
  PdnnSoftmaxParams p = {};
  p.channels = (int)channels;
  p.batch = (int)batch;
  p.rows = (int)rows;
  p.cols = (int)cols;
  const int dtype = dtype_code(inp);
  call([&] { return pdnn_softmax(gradient.defined() ? 1 : 0, dtype, ptr(inp), ptr(gradient), ptr(out), &p, stream()); });
  return THPVariable_Wrap(out);
}

// (a, b, c) with None for an undefined tensor.
PyObject* triple(const at::Tensor& a, const at::Tensor& b, const at::Tensor& c) {
  PyObject* t = PyTuple_New(3);
  if (t == nullptr) throw PyFailure();
  int i = 0;
  for (const at::Tensor* v : {&a, &b, &c}) {
    PyObject* o = v->defined() ? THPVariable_Wrap(*v) : Py_NewRef(Py_None);
    if (o == nullptr) {
      Py_DECREF(t);
      throw PyFailure();
    }
    PyTuple_SET_ITEM(t, i++, o);
  }
  return t;
}

PyObject* batchnorm_forward(PyObject* const* a) {
  const at::Tensor &inp = tensor(a[0]), &beta = tensor(a[1]), &gamma = tensor(a[2]), &mean = tensor(a[3]),
                   &variance = tensor(a[4]);
  const PdnnBatchNormParams p = params<PdnnBatchNormParams>(a[5]);
  require_cuda(inp, beta, gamma, mean, variance, tensor(a[6]));
  const at::Tensor out = out_or_like(tensor(a[6]), inp);
  at::Tensor rm, rv;
  if (p.is_training) {
    rm = like(mean);
    rv = like(variance);
  }
  const int dtype = dtype_code(inp);
  call([&] {
    return pdnn_batchnorm_forward(dtype, ptr(inp), ptr(beta), ptr(gamma), ptr(mean), ptr(variance), ptr(rm), ptr(rv), ptr(out),
                                  &p, stream());
  });
  return triple(out, rm, rv);
}

PyObject* batchnorm_gradient(PyObject* const* a) {
  const at::Tensor &inp = tensor(a[0]), &gradient = tensor(a[1]), &gamma = tensor(a[2]);
  const PdnnBatchNormParams p = params<PdnnBatchNormParams>(a[3]);
  const at::Tensor &pop_mean = tensor(a[4]), &pop_variance = tensor(a[5]);
  require_cuda(inp, gradient, gamma, pop_mean, pop_variance, tensor(a[6]));
  const at::Tensor out = out_or_like(tensor(a[6]), inp), bg = like(gamma), gg = like(gamma);
  const int dtype = dtype_code(inp);
  call([&] {
    return pdnn_batchnorm_gradient(dtype, ptr(inp), ptr(gradient), ptr(gamma), ptr(pop_mean), ptr(pop_variance), ptr(bg),
                                   ptr(gg), ptr(out), &p, stream());
  });
  return triple(out, bg, gg);
}

// The CPython face of one of the functions above: argument count, C++ exceptions to Python ones.
template <PyObject* (*F)(PyObject* const*), int N>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != N) {
    PyErr_Format(PyExc_TypeError, "expected %d arguments, got %zd", N, n);
    return nullptr;
  }
  HANDLE_TH_ERRORS
  try {
    return F(args);
  } catch (const PyFailure&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

#define ENTRY(name, n) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&entry<name, n>)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {ENTRY(conv2d, 17),
                          ENTRY(depthwise_conv2d, 6),
                          ENTRY(pooling, 5),
                          ENTRY(pooling_max_grad, 7),
                          ENTRY(pointwise, 3),
                          ENTRY(pointwise_grad, 4),
                          ENTRY(bias_add, 5),
                          ENTRY(scale_blend, 5),
                          ENTRY(binaryop, 6),
                          ENTRY(matmul, 10),
                          ENTRY(softmax, 7),
                          ENTRY(batchnorm_forward, 7),
                          ENTRY(batchnorm_gradient, 7),
                          {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_front", "Native half of portdnn_b200.api.", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__front(void) { return PyModule_Create(&kModule); }
