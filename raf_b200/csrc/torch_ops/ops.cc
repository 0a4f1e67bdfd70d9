// raf_b200._ops: the host side of the operators that are called once per step or per tensor, on
// torch tensors.  Through ctypes and Python a call cost 10 us before it reached the C ABI
// (argument conversion, per-tensor checks, stream lookup), several times what a small launch takes.
//
// Every function takes the fast way only: when an argument is anything but what the operator
// expects (another type or device, not contiguous, part of an autograd graph), it returns None and has
// done nothing - the Python caller then runs its own checks, which raise.  A failed C ABI call
// returns its status as an int.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <dlfcn.h>

#include <algorithm>
#include <vector>

#include "../../../include/raf_b200.h"

namespace {

// The C ABI of the library that the package has loaded (it need not be the one beside this
// module): bind(path) looks the functions up.
struct {
  decltype(&rafb200_sgd_to) sgd_to;
  decltype(&rafb200_sgd_many) sgd_many;
  decltype(&rafb200_lans_many) lans_many;
  decltype(&rafb200_group_cast) group_cast;
  decltype(&rafb200_fuse_tensor) fuse_tensor;
  decltype(&rafb200_defuse_tensor) defuse_tensor;
} abi;

PyObject* bind(PyObject*, PyObject* path) {
  const char* p = PyUnicode_AsUTF8(path);
  if (!p) return nullptr;
  void* lib = dlopen(p, RTLD_NOW | RTLD_NOLOAD);
  if (!lib) return PyErr_Format(PyExc_ImportError, "%s is not loaded", p);
  auto find = [&](auto& fn, const char* name) {
    fn = reinterpret_cast<std::remove_reference_t<decltype(fn)>>(dlsym(lib, name));
    if (!fn) PyErr_Format(PyExc_ImportError, "%s has no %s", p, name);
    return fn != nullptr;
  };
  if (!find(abi.sgd_to, "rafb200_sgd_to") || !find(abi.sgd_many, "rafb200_sgd_many") ||
      !find(abi.lans_many, "rafb200_lans_many") ||
      !find(abi.group_cast, "rafb200_group_cast") || !find(abi.fuse_tensor, "rafb200_fuse_tensor") ||
      !find(abi.defuse_tensor, "rafb200_defuse_tensor"))
    return nullptr;
  Py_RETURN_NONE;
}

int code_of(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return RAFB200_F32;
    case at::kHalf: return RAFB200_F16;
    case at::kBFloat16: return RAFB200_BF16;
    default: return -1;
  }
}

// Tensors that stand for something else than the values at their address: fake and functional
// ones, subclasses with a dispatch of their own, vmap's batches, lazy negation.
const c10::DispatchKeySet kWrapped({c10::DispatchKey::Python, c10::DispatchKey::Functionalize, c10::DispatchKey::Negative,
                                    c10::DispatchKey::ZeroTensor, c10::DispatchKey::FuncTorchBatched,
                                    c10::DispatchKey::FuncTorchGradWrapper});

// A dense CUDA tensor on the current device (torch.Tensor or Parameter itself: what torch's own calls make
// of a subclass is of that class), or nullptr.  `device` is -1 until the first CUDA tensor
// is met: without a GPU asking for the current device throws, and tensors of the CPU are to be refused
// by the caller's own checks.
const at::Tensor* plain(PyObject* o, c10::DeviceIndex& device) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || t.layout() != at::kStrided || !t.is_cuda() || t.key_set().has_any(kWrapped)) return nullptr;
  if (device < 0) device = c10::cuda::current_device();
  return t.device().index() == device && t.is_contiguous() ? &t : nullptr;
}

// The same where the result belongs to no autograd graph, forward mode included.
const at::Tensor* data_only(PyObject* o, c10::DeviceIndex& device) {
  const at::Tensor* t = plain(o, device);
  return t && !(t->requires_grad() && c10::GradMode::is_enabled()) && !t->_fw_grad(0).defined() ? t : nullptr;
}

void* current_stream(c10::DeviceIndex device) { return c10::cuda::getCurrentCUDAStream(device).stream(); }

PyObject* nothing() { Py_RETURN_NONE; }

// The GIL is released while a function allocates and launches: either may block (the allocator frees its
// cache, a launch queue is full) on something that another Python thread has to bring about.  Tensors that
// are looked at meanwhile are the caller's arguments or held by the call.
struct NoGil {
  PyThreadState* state = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(state); }
  NoGil() = default;
  NoGil(const NoGil&) = delete;
  NoGil& operator=(const NoGil&) = delete;
};

// torch.empty on the current device, from torch's caching allocator: 0.5 us where the dispatched
// form takes 1.3 us, and the list operators make up to hundreds of tensors a call.
at::Tensor new_tensor(at::IntArrayRef sizes, at::ScalarType type) {
  int64_t numel = 1;
  for (int64_t d : sizes) numel *= d;
  const int64_t bytes = numel * (int64_t)c10::elementSize(type);
  c10::Allocator* alloc = c10::cuda::CUDACachingAllocator::get();
  auto storage = c10::make_intrusive<c10::StorageImpl>(c10::StorageImpl::use_byte_size_t(), bytes,
                                                       alloc->allocate((size_t)bytes), alloc, /*resizable=*/true);
  at::Tensor t = at::detail::make_tensor_base<c10::TensorImpl>(std::move(storage), c10::DispatchKeySet(c10::DispatchKey::CUDA),
                                                               c10::scalarTypeToTypeMeta(type));
  t.unsafeGetTensorImpl()->set_sizes_contiguous(sizes);
  return t;
}
// torch.empty_like of a dense tensor: strides of dimensions of one element are kept as they are (a 1x1
// convolution weight in channels_last).
at::Tensor new_like(const at::Tensor& x, at::ScalarType type) {
  at::Tensor t = new_tensor(x.sizes(), type);
  if (x.strides() != t.strides() && x.numel() > 0)  // setting them takes 0.03 us, which 48 tensors show
    t.unsafeGetTensorImpl()->set_sizes_and_strides(x.sizes(), x.strides());
  return t;
}

// sgd(x, dx, v, learning_rate, mu) -> (v1, x1)
PyObject* sgd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 5) return nothing();
  c10::DeviceIndex dev = -1;
  const at::Tensor *x = data_only(a[0], dev), *dx = data_only(a[1], dev), *v = data_only(a[2], dev);
  if (!x || !dx || !v) return nothing();
  const int code = code_of(dx->scalar_type());
  const double lr = PyFloat_AsDouble(a[3]), mu = PyFloat_AsDouble(a[4]);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    return nothing();
  }
  if (x->scalar_type() != at::kFloat || v->scalar_type() != at::kFloat || code < 0 || x->sizes() != dx->sizes() ||
      x->sizes() != v->sizes())
    return nothing();
  at::Tensor x1, v1;
  int rc;
  {
    NoGil released;
    x1 = new_like(*x, at::kFloat);
    v1 = new_like(*v, at::kFloat);
    rc = abi.sgd_to(x->const_data_ptr<float>(), dx->const_data_ptr(), code, v->const_data_ptr<float>(),
                    x1.mutable_data_ptr<float>(), v1.mutable_data_ptr<float>(), x->numel(), (float)lr, (float)mu,
                    current_stream(dev));
  }
  if (rc != RAFB200_OK) return PyLong_FromLong(rc);
  PyObject* out = PyTuple_New(2);
  if (!out) return nullptr;
  PyTuple_SET_ITEM(out, 0, THPVariable_Wrap(std::move(v1)));
  PyTuple_SET_ITEM(out, 1, THPVariable_Wrap(std::move(x1)));
  return out;
}

// Do the byte ranges overlap anywhere, ranges that are only read among themselves excepted?
struct Range {
  uintptr_t lo, hi;
  bool written;
};
bool overlap(std::vector<Range>& r) {
  std::sort(r.begin(), r.end(), [](const Range& p, const Range& q) { return p.lo < q.lo; });
  uintptr_t any = 0, written = 0;  // the furthest ends so far
  for (const Range& x : r) {
    if (x.lo == x.hi) continue;
    if (x.lo < (x.written ? any : written)) return true;
    any = std::max(any, x.hi);
    if (x.written) written = std::max(written, x.hi);
  }
  return false;
}

// sgd_step([(x, v), ...], learning_rate, mu) -> True: every x with a gradient updated in place, one
// launch for all of them.
PyObject* sgd_step(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 3 || !PyList_CheckExact(a[0])) return nothing();
  c10::DeviceIndex dev = -1;
  const double lr = PyFloat_AsDouble(a[1]), mu = PyFloat_AsDouble(a[2]);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    return nothing();
  }
  const Py_ssize_t k = PyList_GET_SIZE(a[0]);
  std::vector<float*> xs, vs;
  std::vector<const void*> gs;
  std::vector<int64_t> numel;
  std::vector<Range> ranges;
  xs.reserve(k);
  vs.reserve(k);
  gs.reserve(k);
  numel.reserve(k);
  ranges.reserve(3 * k);
  int code = -1;
  for (Py_ssize_t i = 0; i < k; ++i) {
    PyObject* pair = PyList_GET_ITEM(a[0], i);
    if (!PyTuple_CheckExact(pair) || PyTuple_GET_SIZE(pair) != 2) return nothing();
    const at::Tensor *x = plain(PyTuple_GET_ITEM(pair, 0), dev), *v = plain(PyTuple_GET_ITEM(pair, 1), dev);
    if (!x || !v) return nothing();
    const at::Tensor& g = x->grad();
    if (!g.defined()) continue;
    const int c = code_of(g.scalar_type());
    if (g.layout() != at::kStrided || !g.is_cuda() || g.device() != x->device() || !g.is_contiguous() || g.key_set().has_any(kWrapped) || c < 0 ||
        (code >= 0 && c != code) || x->scalar_type() != at::kFloat || v->scalar_type() != at::kFloat ||
        g.numel() != x->numel() || v->numel() != x->numel() || x->numel() >= (int64_t(1) << 31))
      return nothing();
    code = c;
    const int64_t ne = x->numel();
    float* xp = static_cast<float*>(x->data_ptr());
    float* vp = static_cast<float*>(v->data_ptr());
    const void* gp = g.const_data_ptr();
    xs.push_back(xp);
    vs.push_back(vp);
    gs.push_back(gp);
    numel.push_back(ne);
    const uintptr_t xb = reinterpret_cast<uintptr_t>(xp), vb = reinterpret_cast<uintptr_t>(vp),
                    gb = reinterpret_cast<uintptr_t>(gp);
    ranges.push_back({xb, xb + ne * 4, true});
    ranges.push_back({vb, vb + ne * 4, true});
    ranges.push_back({gb, gb + ne * g.element_size(), false});
  }
  if (overlap(ranges)) return nothing();  // tied parameters: one after the other, as the loop does
  if (!xs.empty()) {
    int rc;
    {
      NoGil released;
      rc = abi.sgd_many((int)xs.size(), xs.data(), gs.data(), code, vs.data(), numel.data(), (float)lr, (float)mu,
                        current_stream(dev));
    }
    if (rc != RAFB200_OK) return PyLong_FromLong(rc);
  }
  Py_RETURN_TRUE;
}

// lans(tensors, step, learning_rate, beta1, beta2, eps, bias_correction, weight_decay, grad_averaging,
// mode, normalize_grad) -> True: tensors = g + p + m + v, all fp32, p, m and v updated in place.
PyObject* lans(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 11 || !PyList_CheckExact(a[0]) || !PyLong_Check(a[1])) return nothing();
  const Py_ssize_t count = PyList_GET_SIZE(a[0]), k = count / 4;
  if (count == 0 || count % 4 != 0 || k > 0x7fffffff) return nothing();
  const long step = PyLong_AsLong(a[1]), bias_correction = PyLong_AsLong(a[6]), averaging = PyLong_AsLong(a[8]),
             mode = PyLong_AsLong(a[9]);
  const double lr = PyFloat_AsDouble(a[2]), beta1 = PyFloat_AsDouble(a[3]), beta2 = PyFloat_AsDouble(a[4]),
               eps = PyFloat_AsDouble(a[5]), wd = PyFloat_AsDouble(a[7]);
  const int normalize = PyObject_IsTrue(a[10]);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    return nothing();
  }
  if (step < 1 || step > 0x7fffffff || (mode != 0 && mode != 1) || normalize < 0) return nothing();
  c10::DeviceIndex dev = -1;
  std::vector<float*> ptr(count);
  std::vector<int64_t> numel(k);
  std::vector<Range> ranges(count);
  for (Py_ssize_t i = 0; i < count; ++i) {
    const at::Tensor* t = plain(PyList_GET_ITEM(a[0], i), dev);
    if (!t || t->scalar_type() != at::kFloat || t->numel() >= (int64_t(1) << 31)) return nothing();
    if (i < k) numel[i] = t->numel();
    if (t->numel() != numel[i % k]) return nothing();
    ptr[i] = static_cast<float*>(t->data_ptr());
    const uintptr_t at_byte = reinterpret_cast<uintptr_t>(ptr[i]);
    ranges[i] = {at_byte, at_byte + 4 * (uintptr_t)t->numel(), i >= k};
  }
  if (overlap(ranges)) return nothing();
  const size_t bytes = 32 * 512;
  int rc;
  {
    NoGil released;
    c10::DataPtr workspace = c10::cuda::CUDACachingAllocator::get()->allocate(bytes);
    rc = abi.lans_many((int)k, ptr.data(), ptr.data() + k, ptr.data() + 2 * k, ptr.data() + 3 * k, numel.data(), (int)step,
                       (float)lr, (float)beta1, (float)beta2, (float)eps, (int)bias_correction, (float)wd, (int)averaging,
                       (int)mode, normalize, 1.0f, workspace.get(), bytes, current_stream(dev));
  }
  if (rc != RAFB200_OK) return PyLong_FromLong(rc);
  Py_RETURN_TRUE;
}

// The stream argument of an operator: an address, or None for the current stream.
bool stream_of(PyObject* o, c10::DeviceIndex device, void** stream) {
  if (o == Py_None) {
    *stream = current_stream(device);
    return true;
  }
  *stream = PyLong_AsVoidPtr(o);
  if (!PyErr_Occurred()) return true;
  PyErr_Clear();
  return false;
}

// A non-empty list or tuple of dense CUDA tensors of one type: addresses and element counts.  The items are
// held by references of this call (made and given up under the GIL): another thread may change the list.
struct TensorRow {
  std::vector<const at::Tensor*> t;
  std::vector<const void*> ptr;
  std::vector<int64_t> numel;
  std::vector<PyObject*> held;
  TensorRow() = default;
  TensorRow(const TensorRow&) = delete;
  TensorRow& operator=(const TensorRow&) = delete;
  ~TensorRow() {
    for (PyObject* o : held) Py_DECREF(o);
  }
  bool take(PyObject* seq, c10::DeviceIndex& device) {
    if (!PyList_CheckExact(seq) && !PyTuple_CheckExact(seq)) return false;
    const Py_ssize_t k = PySequence_Fast_GET_SIZE(seq);
    PyObject** items = PySequence_Fast_ITEMS(seq);
    t.reserve(k);
    ptr.reserve(k);
    numel.reserve(k);
    held.reserve(k);
    for (Py_ssize_t i = 0; i < k; ++i) {
      const at::Tensor* x = plain(items[i], device);
      if (!x || x->scalar_type() != (i ? t[0] : x)->scalar_type()) return false;
      held.push_back(Py_NewRef(items[i]));
      t.push_back(x);
      ptr.push_back(x->const_data_ptr());
      numel.push_back(x->numel());
    }
    return k > 0;
  }
};

PyObject* wrapped_list(std::vector<at::Tensor>& ts) {
  PyObject* out = PyList_New((Py_ssize_t)ts.size());
  if (!out) return nullptr;
  for (size_t i = 0; i < ts.size(); ++i) PyList_SET_ITEM(out, (Py_ssize_t)i, THPVariable_Wrap(std::move(ts[i])));
  return out;
}

// group_cast(tensors, dtype code, stream) -> list
PyObject* group_cast(PyObject*, PyObject* const* a, Py_ssize_t n) {
  static const at::ScalarType types[] = {at::kFloat, at::kHalf, at::kBFloat16};
  if (n != 3) return nothing();
  c10::DeviceIndex dev = -1;
  TensorRow in;
  void* stream = nullptr;
  const long to = PyLong_AsLong(a[1]);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    return nothing();
  }
  if (to < 0 || to > 2 || !in.take(a[0], dev) || code_of(in.t[0]->scalar_type()) < 0 || !stream_of(a[2], dev, &stream))
    return nothing();
  std::vector<at::Tensor> outs;
  std::vector<void*> dst;
  outs.reserve(in.t.size());
  dst.reserve(in.t.size());
  int rc;
  {
    NoGil released;
    for (const at::Tensor* x : in.t) {
      outs.push_back(new_like(*x, types[to]));
      dst.push_back(outs.back().mutable_data_ptr());
    }
    rc = abi.group_cast((int)in.t.size(), in.ptr.data(), code_of(in.t[0]->scalar_type()), dst.data(), (int)to,
                        in.numel.data(), stream);
  }
  if (rc != RAFB200_OK) return PyLong_FromLong(rc);
  return wrapped_list(outs);
}

// fuse_tensor(tensors, stream) -> flat tensor
PyObject* fuse_tensor(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 2) return nothing();
  c10::DeviceIndex dev = -1;
  TensorRow in;
  void* stream = nullptr;
  if (!in.take(a[0], dev) || !stream_of(a[1], dev, &stream)) return nothing();
  std::vector<int64_t> at_elem(in.t.size());
  int64_t total = 0;
  for (size_t i = 0; i < in.t.size(); ++i) {
    at_elem[i] = total;
    total += in.numel[i];
  }
  at::Tensor flat;
  int rc;
  {
    NoGil released;
    flat = new_tensor({total}, in.t[0]->scalar_type());
    rc = abi.fuse_tensor((int)in.t.size(), in.ptr.data(), in.numel.data(), at_elem.data(), (int)in.t[0]->element_size(),
                         flat.mutable_data_ptr(), stream);
  }
  if (rc != RAFB200_OK) return PyLong_FromLong(rc);
  return THPVariable_Wrap(std::move(flat));
}

bool ints_of(PyObject* seq, std::vector<int64_t>* out) {
  if (!PyList_CheckExact(seq) && !PyTuple_CheckExact(seq)) return false;
  const Py_ssize_t k = PySequence_Fast_GET_SIZE(seq);
  PyObject** items = PySequence_Fast_ITEMS(seq);
  out->resize(k);
  for (Py_ssize_t i = 0; i < k; ++i) {
    if (!PyLong_CheckExact(items[i])) return false;
    (*out)[i] = PyLong_AsLongLong(items[i]);
    if ((*out)[i] < 0) {
      PyErr_Clear();
      return false;
    }
  }
  return true;
}

// defuse_tensor(flat, sizes, shapes, shape_indices, stream) -> list
PyObject* defuse_tensor(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 5) return nothing();
  c10::DeviceIndex dev = -1;
  const at::Tensor* flat = plain(a[0], dev);
  std::vector<int64_t> sizes, dims, ends, at_elem;
  void* stream = nullptr;
  if (!flat || !ints_of(a[1], &sizes) || !ints_of(a[2], &dims) || !ints_of(a[3], &ends) || ends.size() != sizes.size() ||
      !stream_of(a[4], dev, &stream))
    return nothing();
  int64_t total = 0, from = 0;
  for (size_t i = 0; i < sizes.size(); ++i) {
    if (ends[i] < from || ends[i] > (int64_t)dims.size()) return nothing();
    int64_t numel = 1;
    for (int64_t d = from; d < ends[i]; ++d)  // torch.empty refuses what 64 bits cannot count
      if (__builtin_mul_overflow(numel, dims[d], &numel)) return nothing();
    if (numel != sizes[i] || numel > flat->numel() - total) return nothing();
    at_elem.push_back(total);
    total += sizes[i];
    from = ends[i];
  }
  if (sizes.empty()) return nothing();
  std::vector<at::Tensor> outs;
  std::vector<void*> dst;
  outs.reserve(sizes.size());
  dst.reserve(sizes.size());
  from = 0;
  int rc;
  {
    NoGil released;
    for (size_t i = 0; i < sizes.size(); ++i) {
      outs.push_back(new_tensor(at::IntArrayRef(dims.data() + from, (size_t)(ends[i] - from)), flat->scalar_type()));
      dst.push_back(outs.back().mutable_data_ptr());
      from = ends[i];
    }
    rc = abi.defuse_tensor((int)sizes.size(), dst.data(), sizes.data(), at_elem.data(), (int)flat->element_size(),
                           flat->const_data_ptr(), stream);
  }
  if (rc != RAFB200_OK) return PyLong_FromLong(rc);
  return wrapped_list(outs);
}

using Fast = PyObject* (*)(PyObject*, PyObject* const*, Py_ssize_t);

// A C++ exception (the allocator out of memory, first of all) becomes the Python exception that
// torch raises for it; through a plain C entry it would end the process.
template <Fast F>
PyObject* guarded(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  // under a dispatch mode torch's own calls of the slow way are what the mode gets to see
  if (c10::impl::TorchDispatchModeTLS::any_modes_set()) return nothing();
  return F(self, a, n);
  END_HANDLE_TH_ERRORS
}
template <Fast F>
PyCFunction fast() {
  return reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&guarded<F>));
}

PyMethodDef kMethods[] = {
    {"bind", bind, METH_O, "use the C ABI of the loaded library at this path"},
    {"sgd", fast<sgd>(), METH_FASTCALL, "raf.op.sgd"},
    {"sgd_step", fast<sgd_step>(), METH_FASTCALL, "eager SGD, all parameters"},
    {"lans", fast<lans>(), METH_FASTCALL, "raf.op.lans"},
    {"group_cast", fast<group_cast>(), METH_FASTCALL, "raf.op.group_cast"},
    {"fuse_tensor", fast<fuse_tensor>(), METH_FASTCALL, "raf.op.fuse_tensor"},
    {"defuse_tensor", fast<defuse_tensor>(), METH_FASTCALL,
     "raf.op.defuse_tensor"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_ops", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__ops() { return PyModule_Create(&kModule); }
