// Host side of the Python mirror: the C ABI's entry points as Python functions that take torch tensors.
//
// What bounds a small call is the host. Through ctypes an entry point with twenty arguments cost 4 to 6 us of
// argument objects before its kernel launch (2.1 us), and the shape arithmetic and allocations of the Python
// mirror as much again. Here each argument is read straight from its Python object by the parameter's C type, the
// device and stream come from the tensors, and the helpers below do the mirror's per-call checks and allocations.
// Measured per call, before and after, with the launch: ReLU of a small tensor 8.2 -> 4.7 us, a binary-weight
// convolution 21.8 -> 8.1 us, a folded convolution 23.4 -> 4.3 us.
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <algorithm>
#include <array>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <tuple>
#include <type_traits>
#include <utility>
#include <vector>

#include "nnabla_b200.h"

namespace {

std::atomic<long long> g_calls{0};

// nnabla_b200._capi.NB200Error(code, message)
PyObject *raise_status(int code) {
  static PyObject *cls = nullptr; // (the GIL is held)
  if (!cls) {
    PyObject *m = PyImport_ImportModule("nnabla_b200._capi");
    if (!m)
      return nullptr;
    cls = PyObject_GetAttrString(m, "NB200Error");
    Py_DECREF(m);
    if (!cls)
      return nullptr;
  }
  const char *text = nb200_last_error();
  PyObject *e = PyObject_CallFunction(cls, "iN", code, PyUnicode_DecodeUTF8(text, (Py_ssize_t)strlen(text), "replace"));
  if (e) {
    PyErr_SetObject(cls, e);
    Py_DECREF(e);
  }
  return nullptr;
}

// ---- arguments ----------------------------------------------------------------------------------------------------
constexpr int kMaxExtents = 16; // of a shape passed as a tuple

// One argument of C type T read from a Python object. `device` receives the index of the first CUDA tensor seen.
template <typename T, typename Enable = void> struct Arg;

template <typename T> struct Arg<T, std::enable_if_t<std::is_integral_v<T>>> {
  T v;
  bool read(PyObject *o, int &) {
    long long n = PyLong_AsLongLong(o);
    if (n == -1 && PyErr_Occurred()) {
      PyErr_Clear();
      PyObject *i = PyNumber_Long(o); // what int(o) accepts
      if (!i)
        return false;
      n = PyLong_AsLongLong(i);
      Py_DECREF(i);
      if (n == -1 && PyErr_Occurred())
        return false;
    }
    v = (T)n;
    return true;
  }
};

template <> struct Arg<float> {
  float v;
  bool read(PyObject *o, int &) {
    const double d = PyFloat_AsDouble(o);
    v = (float)d;
    return !(d == -1.0 && PyErr_Occurred());
  }
};

template <typename P> struct Arg<P *> {
  using E = std::remove_const_t<P>;
  static constexpr bool kShape = std::is_same_v<P, const int64_t> || std::is_same_v<P, const int>;
  P *v;
  std::array<std::conditional_t<kShape, E, char>, kShape ? kMaxExtents : 1> buf;
  bool read(PyObject *o, int &device) {
    if (o == Py_None) {
      v = nullptr;
      return true;
    }
    if (THPVariable_Check(o)) {
      const at::Tensor &t = THPVariable_Unpack(o);
      if (device < 0 && t.is_cuda())
        device = t.get_device();
      v = static_cast<P *>(t.data_ptr());
      return true;
    }
    if constexpr (kShape) {
      if (PyTuple_Check(o) || PyList_Check(o)) {
        const Py_ssize_t n = PySequence_Fast_GET_SIZE(o);
        if (n > kMaxExtents) {
          PyErr_Format(PyExc_RuntimeError, "more than %d extents", kMaxExtents);
          return false;
        }
        for (Py_ssize_t i = 0; i < n; ++i) {
          Arg<E> a;
          if (!a.read(PySequence_Fast_GET_ITEM(o, i), device))
            return false;
          buf[i] = a.v;
        }
        v = buf.data();
        return true;
      }
    }
    if (PyLong_Check(o)) {
      v = static_cast<P *>(PyLong_AsVoidPtr(o));
      return !PyErr_Occurred();
    }
    PyErr_Format(PyExc_TypeError, "expected a tensor, None or an address, got %s", Py_TYPE(o)->tp_name);
    return false;
  }
};

template <typename Tuple, size_t... I>
bool read_args(Tuple &a, PyObject *const *args, int &device, std::index_sequence<I...>) {
  return (std::get<I>(a).read(args[I], device) && ...);
}

// Makes `device` the current one, and the caller's again on every way out of the block, exceptions among them.
class OnDevice {
  const int device_, before_;

public:
  explicit OnDevice(int device) : device_(device), before_(c10::cuda::current_device()) {
    if (device_ != before_)
      c10::cuda::set_device((c10::DeviceIndex)device_);
  }
  ~OnDevice() {
    if (device_ != before_)
      (void)c10::cuda::SetDevice((c10::DeviceIndex)before_); // (the one of the two that does not throw)
  }
  OnDevice(const OnDevice &) = delete;
  OnDevice &operator=(const OnDevice &) = delete;
};

// The entry point as a Python function of its parameters without the last one, `stream`: that is torch's current
// stream of the tensors' device, which is made the current device for the call.
template <auto Fn> struct Entry;
template <typename... A, int (*Fn)(A...)> struct Entry<Fn> {
  static PyObject *call(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    constexpr size_t n = sizeof...(A) - 1;
    if (nargs != (Py_ssize_t)n)
      return PyErr_Format(PyExc_TypeError, "expected %zu arguments, got %zd", n, nargs);
    std::tuple<Arg<A>...> a;
    int device = -1;
    if (!read_args(a, args, device, std::make_index_sequence<n>{}))
      return nullptr;
    if (device < 0) // (no tensor among the arguments)
      device = c10::cuda::current_device();
    const OnDevice on(device);
    std::get<n>(a).v = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream();
    g_calls.fetch_add(1, std::memory_order_relaxed);
    int rc;
    Py_BEGIN_ALLOW_THREADS;
    rc = std::apply([](auto &...x) { return Fn(x.v...); }, a);
    Py_END_ALLOW_THREADS;
    if (rc != 0)
      return raise_status(rc);
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
  }
};

// ---- the mirror's per-call checks and allocations ------------------------------------------------------------------
PyObject *calls(PyObject *, PyObject *) { return PyLong_FromLongLong(g_calls.load(std::memory_order_relaxed)); }

bool plain_f32(PyObject *o) {
  if (!THPVariable_Check(o))
    return false;
  const at::Tensor &t = THPVariable_Unpack(o);
  return t.is_cuda() && t.scalar_type() == at::kFloat && t.is_contiguous();
}

// f32(x, name="x"): x if it is a contiguous float32 CUDA tensor, a contiguous copy if it is not contiguous; an
// exception otherwise.
PyObject *f32(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs < 1 || nargs > 2)
    return PyErr_Format(PyExc_TypeError, "expected 1 or 2 arguments, got %zd", nargs);
  PyObject *o = args[0];
  if (plain_f32(o)) {
    Py_INCREF(o);
    return o;
  }
  const char *name = nargs > 1 ? PyUnicode_AsUTF8(args[1]) : "x";
  if (!name)
    return nullptr;
  if (!THPVariable_Check(o))
    return PyErr_Format(PyExc_TypeError, "%s must be a torch.Tensor on a CUDA device", name);
  const at::Tensor &t = THPVariable_Unpack(o);
  if (!t.is_cuda())
    return PyErr_Format(PyExc_RuntimeError, "nnabla_b200 has no CPU path: %s is on %s", name, t.device().str().c_str());
  if (t.scalar_type() != at::kFloat) {
    PyObject *dtype = PyObject_GetAttrString(o, "dtype");
    if (dtype) {
      PyErr_Format(PyExc_TypeError, "%s must be float32 (the 'float' type config), got %S", name, dtype);
      Py_DECREF(dtype);
    }
    return nullptr;
  }
  return THPVariable_Wrap(t.contiguous());
  END_HANDLE_TH_ERRORS
}

bool read_shape(PyObject *o, c10::SmallVector<int64_t, 8> &out) {
  if (THPVariable_Check(o)) {
    const at::IntArrayRef s = THPVariable_Unpack(o).sizes();
    out.assign(s.begin(), s.end());
    return true;
  }
  if (!PyTuple_Check(o) && !PyList_Check(o)) {
    PyErr_SetString(PyExc_TypeError, "a shape is a tensor's, a tuple or a list");
    return false;
  }
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(o);
  int unused = 0;
  for (Py_ssize_t i = 0; i < n; ++i) {
    Arg<int64_t> a;
    if (!a.read(PySequence_Fast_GET_ITEM(o, i), unused))
      return false;
    out.push_back(a.v);
  }
  return true;
}

// empty(shape, like) / empty_i8(shape, like): an uninitialised tensor of `shape` on the device of `like`.
template <at::ScalarType kType> PyObject *empty(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 2 || !THPVariable_Check(args[1]))
    return PyErr_Format(PyExc_TypeError, "expected a shape and a tensor");
  c10::SmallVector<int64_t, 8> shape;
  if (!read_shape(args[0], shape))
    return nullptr;
  return THPVariable_Wrap(at::detail::empty_cuda(at::IntArrayRef(shape.data(), shape.size()), kType,
                                                 THPVariable_Unpack(args[1]).device(), std::nullopt));
  END_HANDLE_TH_ERRORS
}

bool read_pair(PyObject *o, int64_t fallback, int64_t out[2]) {
  if (o == Py_None) {
    out[0] = out[1] = fallback;
    return true;
  }
  if (!PyTuple_Check(o) && !PyList_Check(o))
    return false;
  if (PySequence_Fast_GET_SIZE(o) != 2)
    return false;
  for (int i = 0; i < 2; ++i) {
    PyObject *e = PySequence_Fast_GET_ITEM(o, i);
    if (!PyLong_Check(e))
      return false;
    out[i] = PyLong_AsLongLong(e);
  }
  return !PyErr_Occurred();
}

// Geometry of a 2-D convolution with one batch axis; false where the operands do not fit together.
struct Geometry {
  int64_t x[4], w[4], pad[2], stride[2], dil[2], out[2];
  bool read(const c10::SmallVector<int64_t, 8> &xs, const c10::SmallVector<int64_t, 8> &ws, PyObject *p, PyObject *st,
            PyObject *d, long group) {
    if (xs.size() != 4 || ws.size() != 4 || group <= 0)
      return false;
    std::copy(xs.begin(), xs.end(), x);
    std::copy(ws.begin(), ws.end(), w);
    bool ok = read_pair(p, 0, pad) && read_pair(st, 1, stride) && read_pair(d, 1, dil) && x[1] % group == 0 &&
              w[0] % group == 0 && x[1] / group == w[1];
    for (int i = 0; ok && i < 2; ++i) {
      const int64_t span = x[2 + i] + 2 * pad[i] - (dil[i] * (w[2 + i] - 1) + 1);
      ok = span >= 0 && stride[i] > 0;
      out[i] = ok ? span / stride[i] + 1 : 0;
    }
    if (!ok)
      PyErr_Clear();
    return ok;
  }
};

// conv2d(x, w, bias, base_axis, pad, stride, dilation, group): the geometry of a 2-D convolution with one batch axis,
// (batch, channels, height, width, outmaps, kh, kw, pad, stride, dilation, output shape); x and w are tensors or
// shapes. None where the operands are of another form or do not fit together: the caller's full checks say why.
PyObject *conv2d(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 8)
    return PyErr_Format(PyExc_TypeError, "expected 8 arguments, got %zd", nargs);
  c10::SmallVector<int64_t, 8> x, w, b;
  Geometry g;
  const long base_axis = PyLong_AsLong(args[3]), group = PyLong_AsLong(args[7]);
  bool ok = !PyErr_Occurred() && base_axis == 1 && read_shape(args[0], x) && read_shape(args[1], w) &&
            g.read(x, w, args[4], args[5], args[6], group);
  if (ok && args[2] != Py_None)
    ok = read_shape(args[2], b) && b.size() == 1 && b[0] == w[0];
  if (!ok) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  return Py_BuildValue("LLLLLLL(LL)(LL)(LL)(LLLL)", (long long)x[0], (long long)x[1], (long long)x[2], (long long)x[3],
                       (long long)w[0], (long long)w[2], (long long)w[3], (long long)g.pad[0], (long long)g.pad[1],
                       (long long)g.stride[0], (long long)g.stride[1], (long long)g.dil[0], (long long)g.dil[1],
                       (long long)x[0], (long long)w[0], (long long)g.out[0], (long long)g.out[1]);
  END_HANDLE_TH_ERRORS
}

PyObject *codes_nhwc_slots(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  Arg<int64_t> channels;
  Arg<int> group;
  int unused = 0;
  if (nargs != 2 || !channels.read(args[0], unused) || !group.read(args[1], unused))
    return PyErr_Occurred() ? nullptr : PyErr_Format(PyExc_TypeError, "expected channels and group");
  return PyLong_FromLongLong(nb200_codes_nhwc_slots(channels.v, group.v));
  END_HANDLE_TH_ERRORS
}

// ---- whole calls of the mirror -------------------------------------------------------------------------------------
// The functions that networks and training blocks call per layer, from their Python arguments to the launch: checks,
// geometry and allocations in Python cost a folded convolution 3.9 us on top of 3.3. Each returns None, before anything
// is written or launched, where an argument is not of the plain form; the caller's full path then does the work or says
// what is wrong.

// Tensors, shapes and options of one call; ok turns false at the first that is not of the plain form.
struct Plain {
  bool ok = true;
  const at::Tensor *first = nullptr;
  // a contiguous float32 CUDA tensor on the device of the first one
  const at::Tensor *f32(PyObject *o) { return tensor(o, at::kFloat); }
  const at::Tensor *i8(PyObject *o) { return tensor(o, at::kChar); }
  const at::Tensor *tensor(PyObject *o, at::ScalarType type) {
    if (!ok || !THPVariable_Check(o))
      return fail();
    const at::Tensor &t = THPVariable_Unpack(o);
    if (!t.is_cuda() || t.scalar_type() != type || !t.is_contiguous() || (first && t.get_device() != first->get_device()))
      return fail();
    if (!first)
      first = &t;
    return &t;
  }
  // the same, or NULL for None
  const at::Tensor *f32_or_none(PyObject *o) { return o == Py_None ? nullptr : f32(o); }
  const at::Tensor *fail() {
    ok = false;
    return nullptr;
  }
  void require(bool condition) { ok = ok && condition; }
  // the truth of a bool; anything else is not plain
  bool truth(PyObject *o) {
    require(o == Py_True || o == Py_False);
    return o == Py_True;
  }
  long integer(PyObject *o) {
    const long v = ok && PyLong_Check(o) ? PyLong_AsLong(o) : (ok = false, 0);
    if (v == -1 && PyErr_Occurred()) {
      PyErr_Clear();
      ok = false;
    }
    return v;
  }
  float number(PyObject *o) {
    if (ok && (PyFloat_Check(o) || PyLong_Check(o))) {
      const double d = PyFloat_AsDouble(o);
      if (!(d == -1.0 && PyErr_Occurred()))
        return (float)d;
      PyErr_Clear();
    }
    ok = false;
    return 0.0f;
  }
};

template <typename P> P *data(const at::Tensor *t) { return t ? static_cast<P *>(t->data_ptr()) : nullptr; }

at::Tensor empty_like_of(const at::Tensor &like, at::IntArrayRef shape, at::ScalarType type) {
  return at::detail::empty_cuda(shape, type, like.device(), std::nullopt);
}

// Runs an entry point on the tensors' device and torch's current stream of it; NULL after raising its error.
template <typename F> bool run_on(const at::Tensor &t, F &&f) {
  const int device = t.get_device();
  const OnDevice on(device);
  void *stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream();
  g_calls.fetch_add(1, std::memory_order_relaxed);
  int rc;
  Py_BEGIN_ALLOW_THREADS;
  rc = f(stream);
  Py_END_ALLOW_THREADS;
  if (rc != 0)
    raise_status(rc);
  return rc == 0;
}

PyObject *not_plain() {
  PyErr_Clear();
  Py_RETURN_NONE;
}

// folded_convolution(x_codes, x_shape, side, group, w_shape, scale, bias, pad, stride, dilation, residual_codes,
//                    residual_delta, residual, relu, sign, n, delta, output): functions.convolution_codes_folded
PyObject *folded_convolution(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 18)
    return PyErr_Format(PyExc_TypeError, "expected 18 arguments, got %zd", nargs);
  Plain p;
  c10::SmallVector<int64_t, 8> xs, ws;
  Geometry g;
  const at::Tensor *x = p.i8(a[0]), *side = p.i8(a[2]), *scale = p.f32(a[5]), *bias = p.f32_or_none(a[6]);
  const at::Tensor *res_codes = a[10] == Py_None ? nullptr : p.i8(a[10]), *res = p.f32_or_none(a[12]);
  const float res_delta = a[11] == Py_None ? 0.0f : p.number(a[11]);
  const bool relu = p.truth(a[13]), sign = p.truth(a[14]);
  const long n = p.integer(a[15]);
  const float delta = p.number(a[16]);
  const char *output = PyUnicode_Check(a[17]) ? PyUnicode_AsUTF8(a[17]) : nullptr;
  const bool codes = output && strcmp(output, "codes") == 0;
  p.require(output && (codes || strcmp(output, "float") == 0) && p.integer(a[3]) == 1);
  if (!p.ok || !read_shape(a[1], xs) || !read_shape(a[4], ws) || !g.read(xs, ws, a[7], a[8], a[9], 1))
    return not_plain();
  const int64_t pixels = g.out[0] * g.out[1], slots = nb200_codes_nhwc_slots(g.w[0], 1);
  const int64_t want_x[3] = {g.x[0], g.x[2] * g.x[3], nb200_codes_nhwc_slots(g.x[1], 1)}, want_y[3] = {g.x[0], pixels, slots};
  const at::IntArrayRef y_shape(want_y, 3);
  p.require(x->sizes() == at::IntArrayRef(want_x, 3) && scale->numel() == g.w[0] &&
            (!bias || (bias->dim() == 1 && bias->numel() == g.w[0])) && (!res_codes || res_codes->sizes() == y_shape) &&
            (!res || res->sizes() == y_shape));
  if (!p.ok)
    return not_plain();
  const at::Tensor y = empty_like_of(*x, y_shape, codes ? at::kChar : at::kFloat);
  if (!run_on(*x, [&](void *stream) {
        return nb200_convolution_codes_folded_nhwc(
            data<int8_t>(x), data<int8_t>(side), data<float>(scale), data<float>(bias), data<int8_t>(res_codes), res_delta,
            data<float>(res), codes ? data<int8_t>(&y) : nullptr, codes ? nullptr : data<float>(&y), (int)g.x[0], (int)g.x[1],
            (int)g.x[2], (int)g.x[3], (int)g.w[0], (int)g.w[2], (int)g.w[3], (int)g.pad[0], (int)g.pad[1],
            (int)g.stride[0], (int)g.stride[1], (int)g.dil[0], (int)g.dil[1], relu, sign, (int)n, delta, stream);
      }))
    return nullptr;
  return Py_BuildValue("N(LLLL)", THPVariable_Wrap(y), (long long)g.x[0], (long long)g.w[0], (long long)g.out[0],
                       (long long)g.out[1]);
  END_HANDLE_TH_ERRORS
}

PyObject *attribute(PyObject *o, const char *name) { // new reference; NULL without an exception
  PyObject *v = PyObject_GetAttrString(o, name);
  if (!v)
    PyErr_Clear();
  return v;
}

// folded_convolutions(x_codes, x_shape, steps, n, delta): functions.folded_convolutions. All steps are read and checked
// before the first is launched.
PyObject *folded_convolutions(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 5)
    return PyErr_Format(PyExc_TypeError, "expected 5 arguments, got %zd", nargs);
  struct Step {
    Geometry g;
    at::Tensor side; // (held: the prepared weights' attribute could be set anew while other threads run)
    const at::Tensor *scale, *bias;
    int64_t source, residual;
    bool relu, codes;
    int64_t last_use; // of its result
  };
  Plain p;
  const at::Tensor *x = p.i8(a[0]);
  c10::SmallVector<int64_t, 8> xs;
  const long n = p.integer(a[3]);
  const float delta = p.number(a[4]);
  if (!p.ok || !read_shape(a[1], xs) || xs.size() != 4 || !PyTuple_Check(a[2]))
    return not_plain();
  const int64_t count = PyTuple_GET_SIZE(a[2]), want_x[3] = {xs[0], xs[2] * xs[3], nb200_codes_nhwc_slots(xs[1], 1)};
  p.require(count > 0 && x->sizes() == at::IntArrayRef(want_x, 3));
  std::vector<Step> steps((size_t)count);
  for (int64_t i = 0; p.ok && i < count; ++i) {
    PyObject *t = PyTuple_GET_ITEM(a[2], i);
    if (!PyTuple_Check(t) || PyTuple_GET_SIZE(t) != 9)
      return not_plain();
    auto item = [&](int k) { return PyTuple_GET_ITEM(t, k); };
    Step &s = steps[(size_t)i];
    s.last_use = i;
    s.source = p.integer(item(0));
    PyObject *prepared = item(1), *side = attribute(prepared, "side"), *shape = attribute(prepared, "shape"),
             *group = attribute(prepared, "group");
    if (const at::Tensor *t8 = side ? p.i8(side) : p.fail())
      s.side = *t8;
    c10::SmallVector<int64_t, 8> in, ws;
    p.require(group && p.integer(group) == 1 && shape && read_shape(shape, ws) && s.source >= 0 && s.source <= i);
    Py_XDECREF(side);
    Py_XDECREF(shape);
    Py_XDECREF(group);
    s.scale = p.f32(item(2)), s.bias = p.f32_or_none(item(3));
    const bool adds = item(6) != Py_None;
    s.residual = adds ? p.integer(item(6)) : -1;
    s.relu = p.truth(item(7)), s.codes = p.truth(item(8));
    p.require(!adds || (s.residual >= 0 && s.residual <= i));
    if (!p.ok)
      return not_plain();
    if (s.source == 0) {
      in = xs;
    } else {
      const Step &from = steps[(size_t)s.source - 1];
      p.require(from.codes);
      in = {from.g.x[0], from.g.w[0], from.g.out[0], from.g.out[1]};
    }
    p.require(s.g.read(in, ws, item(4), item(5), Py_None, 1) && s.scale->numel() == s.g.w[0] &&
              (!s.bias || (s.bias->dim() == 1 && s.bias->numel() == s.g.w[0])));
    if (p.ok && s.residual >= 0) { // of the result's own shape
      const int64_t *o = s.residual == 0 ? xs.data() : nullptr;
      const Step *from = o ? nullptr : &steps[(size_t)s.residual - 1];
      const int64_t r[4] = {o ? o[0] : from->g.x[0], o ? o[1] : from->g.w[0], o ? o[2] : from->g.out[0], o ? o[3] : from->g.out[1]};
      p.require(r[0] == s.g.x[0] && r[1] == s.g.w[0] && r[2] == s.g.out[0] && r[3] == s.g.out[1]);
      if (s.residual > 0)
        steps[(size_t)s.residual - 1].last_use = i;
    }
    if (s.source > 0)
      steps[(size_t)s.source - 1].last_use = i;
  }
  if (!p.ok)
    return not_plain();
  std::vector<at::Tensor> results((size_t)count);
  int rc = 0;
  {
    const int device = x->get_device();
    const OnDevice on(device); // (an allocation below may throw)
    void *stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream();
    pybind11::gil_scoped_release no_gil;
    for (int64_t i = 0; i < count && rc == 0; ++i) {
      const Step &s = steps[(size_t)i];
      const Geometry &g = s.g;
      const int64_t want[3] = {g.x[0], g.out[0] * g.out[1], nb200_codes_nhwc_slots(g.w[0], 1)};
      at::Tensor &y = results[(size_t)i];
      y = empty_like_of(*x, at::IntArrayRef(want, 3), s.codes ? at::kChar : at::kFloat);
      const at::Tensor *from = s.source == 0 ? x : &results[(size_t)s.source - 1];
      const at::Tensor *res = s.residual < 0 ? nullptr : s.residual == 0 ? x : &results[(size_t)s.residual - 1];
      const bool res_codes = res && res->scalar_type() == at::kChar;
      g_calls.fetch_add(1, std::memory_order_relaxed);
      rc = nb200_convolution_codes_folded_nhwc(
          data<int8_t>(from), data<int8_t>(&s.side), data<float>(s.scale), data<float>(s.bias),
          res_codes ? data<int8_t>(res) : nullptr, res_codes ? delta : 0.0f, res_codes ? nullptr : data<float>(res),
          s.codes ? data<int8_t>(&y) : nullptr, s.codes ? nullptr : data<float>(&y), (int)g.x[0], (int)g.x[1], (int)g.x[2],
          (int)g.x[3], (int)g.w[0], (int)g.w[2], (int)g.w[3], (int)g.pad[0], (int)g.pad[1], (int)g.stride[0],
          (int)g.stride[1], (int)g.dil[0], (int)g.dil[1], s.relu, 1, (int)n, delta, stream);
      for (int64_t j = 0; j < i; ++j)
        if (steps[(size_t)j].last_use == i)
          results[(size_t)j].reset();
    }
  }
  if (rc != 0)
    return raise_status(rc);
  const Geometry &g = steps.back().g;
  return Py_BuildValue("N(LLLL)", THPVariable_Wrap(results.back()), (long long)g.x[0], (long long)g.w[0], (long long)g.out[0],
                       (long long)g.out[1]);
  END_HANDLE_TH_ERRORS
}

// binary_convolution(x, weight, binary_weight, alpha, bias, pad, stride, dilation, group, quantize_zero_to, delta):
// y of binary_weight_convolution (alpha a tensor) or binary_connect_convolution (alpha None); delta None or a number
PyObject *binary_convolution(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 11)
    return PyErr_Format(PyExc_TypeError, "expected 11 arguments, got %zd", nargs);
  Plain p;
  c10::SmallVector<int64_t, 8> xs, ws;
  Geometry g;
  const at::Tensor *x = p.f32(a[0]), *w = p.f32(a[1]), *wb = p.f32(a[2]), *alpha = p.f32_or_none(a[3]),
                   *bias = p.f32_or_none(a[4]);
  const long group = p.integer(a[8]);
  const float zero_to = p.number(a[9]), delta = a[10] == Py_None ? 0.0f : p.number(a[10]);
  if (!p.ok || !read_shape(a[0], xs) || !read_shape(a[1], ws) || !g.read(xs, ws, a[5], a[6], a[7], group))
    return not_plain();
  p.require(w->sizes() == wb->sizes() && (!alpha || alpha->numel() == g.w[0]) &&
            (!bias || (bias->dim() == 1 && bias->numel() == g.w[0])));
  if (!p.ok)
    return not_plain();
  const int64_t out[4] = {g.x[0], g.w[0], g.out[0], g.out[1]};
  const at::Tensor y = empty_like_of(*x, at::IntArrayRef(out, 4), at::kFloat);
  const int c[13] = {(int)g.x[0],   (int)g.x[1],   (int)g.x[2],      (int)g.x[3],      (int)g.w[0],   (int)g.w[2],  (int)g.w[3],
                     (int)g.pad[0], (int)g.pad[1], (int)g.stride[0], (int)g.stride[1], (int)g.dil[0], (int)g.dil[1]};
  if (!run_on(*x, [&](void *stream) {
        return alpha ? nb200_binary_weight_convolution_f32(data<float>(x), data<float>(w), data<float>(wb),
                                                           data<float>(alpha), data<float>(bias), data<float>(&y), c[0], c[1],
                                                           c[2], c[3], c[4], c[5], c[6], c[7], c[8], c[9], c[10], c[11],
                                                           c[12], (int)group, zero_to, delta, stream)
                     : nb200_binary_connect_convolution_f32(data<float>(x), data<float>(w), data<float>(wb),
                                                            data<float>(bias), data<float>(&y), c[0], c[1], c[2], c[3], c[4],
                                                            c[5], c[6], c[7], c[8], c[9], c[10], c[11], c[12], (int)group,
                                                            zero_to, delta, stream);
      }))
    return nullptr;
  return THPVariable_Wrap(y);
  END_HANDLE_TH_ERRORS
}

bool read_flags(Plain &p, PyObject *o, bool out[3]) {
  if (!PyTuple_Check(o) || PyTuple_GET_SIZE(o) != 3)
    return p.ok = false;
  for (int i = 0; i < 3; ++i)
    out[i] = p.truth(PyTuple_GET_ITEM(o, i));
  return p.ok;
}

// binary_convolution_backward(x, binary_weight, alpha, dy, pad, stride, dilation, group, propagate_down, accum, grads,
// delta): (dx, dw, db) with what grads holds where propagate_down is False
PyObject *binary_convolution_backward(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 12)
    return PyErr_Format(PyExc_TypeError, "expected 12 arguments, got %zd", nargs);
  Plain p;
  c10::SmallVector<int64_t, 8> xs, ws;
  Geometry g;
  const at::Tensor *x = p.f32(a[0]), *wb = p.f32(a[1]), *alpha = p.f32_or_none(a[2]), *dy = p.f32(a[3]);
  const long group = p.integer(a[7]);
  bool down[3], accum[3];
  read_flags(p, a[8], down);
  read_flags(p, a[9], accum);
  const float delta = a[11] == Py_None ? 0.0f : p.number(a[11]);
  p.require(PyTuple_Check(a[10]) && PyTuple_GET_SIZE(a[10]) == 3);
  if (!p.ok || !read_shape(a[0], xs) || !read_shape(a[1], ws) || !g.read(xs, ws, a[4], a[5], a[6], group))
    return not_plain();
  const int64_t out[4] = {g.x[0], g.w[0], g.out[0], g.out[1]};
  p.require(dy->sizes() == at::IntArrayRef(out, 4));
  const at::IntArrayRef shapes[3] = {x->sizes(), wb->sizes(), at::IntArrayRef(g.w, 1)};
  at::Tensor grad[3];
  for (int i = 0; p.ok && i < 3; ++i) {
    PyObject *given = PyTuple_GET_ITEM(a[10], i);
    if (!down[i])
      continue;
    if (given == Py_None) {
      p.require(!accum[i]);
    } else {
      const at::Tensor *t = p.f32(given);
      p.require(t && t->sizes() == shapes[i]);
      if (p.ok)
        grad[i] = *t;
    }
  }
  if (!p.ok)
    return not_plain();
  for (int i = 0; i < 3; ++i)
    if (down[i] && !grad[i].defined())
      grad[i] = empty_like_of(*x, shapes[i], at::kFloat);
  float *d[3];
  for (int i = 0; i < 3; ++i)
    d[i] = down[i] ? data<float>(&grad[i]) : nullptr;
  const int c[13] = {(int)g.x[0],   (int)g.x[1],   (int)g.x[2],      (int)g.x[3],      (int)g.w[0],   (int)g.w[2],  (int)g.w[3],
                     (int)g.pad[0], (int)g.pad[1], (int)g.stride[0], (int)g.stride[1], (int)g.dil[0], (int)g.dil[1]};
  if (!run_on(*x, [&](void *stream) {
        return alpha ? nb200_binary_weight_convolution_backward_f32(
                           data<float>(x), data<float>(wb), data<float>(alpha), data<float>(dy), d[0], d[1], d[2], c[0], c[1],
                           c[2], c[3], c[4], c[5], c[6], c[7], c[8], c[9], c[10], c[11], c[12], (int)group, accum[0],
                           accum[1], accum[2], delta, stream)
                     : nb200_binary_connect_convolution_backward_f32(
                           data<float>(x), data<float>(wb), data<float>(dy), d[0], d[1], d[2], c[0], c[1], c[2], c[3], c[4],
                           c[5], c[6], c[7], c[8], c[9], c[10], c[11], c[12], (int)group, accum[0], accum[1], accum[2],
                           delta, stream);
      }))
    return nullptr;
  PyObject *r = PyTuple_New(3);
  for (int i = 0; r && i < 3; ++i) {
    PyObject *given = PyTuple_GET_ITEM(a[10], i);
    if (!down[i] || given != Py_None) {
      Py_INCREF(given);
      PyTuple_SET_ITEM(r, i, given);
    } else {
      PyTuple_SET_ITEM(r, i, THPVariable_Wrap(grad[i]));
    }
  }
  return r;
  END_HANDLE_TH_ERRORS
}

// channel axis 1, given as [1] or (1,)
bool axis_one(PyObject *o) {
  if (!(PyList_Check(o) || PyTuple_Check(o)) || PySequence_Fast_GET_SIZE(o) != 1)
    return false;
  PyObject *e = PySequence_Fast_GET_ITEM(o, 0);
  return PyLong_Check(e) && PyLong_AsLong(e) == 1;
}

// batch_normalization(x, beta, gamma, mean, variance, axes, decay_rate, eps, batch_stat, output_stat)
PyObject *batch_normalization(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 10)
    return PyErr_Format(PyExc_TypeError, "expected 10 arguments, got %zd", nargs);
  Plain p;
  const at::Tensor *x = p.f32(a[0]), *beta = p.f32_or_none(a[1]), *gamma = p.f32_or_none(a[2]), *mean = p.f32(a[3]),
                   *var = p.f32(a[4]);
  const float decay = p.number(a[6]), eps = p.number(a[7]);
  const bool batch = p.truth(a[8]), stats = p.truth(a[9]);
  p.require(axis_one(a[5]) && p.ok && x->dim() >= 2);
  if (!p.ok)
    return not_plain();
  const int64_t outer = x->size(0), C = x->size(1), inner = x->numel() / std::max<int64_t>(outer * C, 1);
  for (const at::Tensor *t : {beta, gamma, mean, var})
    p.require(!t || t->numel() == C);
  if (!p.ok)
    return not_plain();
  const at::Tensor y = empty_like_of(*x, x->sizes(), at::kFloat);
  at::Tensor bm, bv;
  if (batch) {
    bm = empty_like_of(*x, mean->sizes(), at::kFloat);
    bv = empty_like_of(*x, var->sizes(), at::kFloat);
  }
  if (!run_on(*x, [&](void *stream) {
        return batch ? nb200_batch_normalization_batch_f32(data<float>(x), data<float>(beta), data<float>(gamma),
                                                           data<float>(mean), data<float>(var), data<float>(&y),
                                                           data<float>(&bm), data<float>(&bv), outer, C, inner, eps, decay, 1,
                                                           stream)
                     : nb200_batch_normalization_inference_f32(data<float>(x), data<float>(beta), data<float>(gamma),
                                                               data<float>(mean), data<float>(var), data<float>(&y), outer,
                                                               C, inner, eps, stream);
      }))
    return nullptr;
  if (batch && stats)
    return Py_BuildValue("NNN", THPVariable_Wrap(y), THPVariable_Wrap(bm), THPVariable_Wrap(bv));
  return THPVariable_Wrap(y);
  END_HANDLE_TH_ERRORS
}

// batch_normalization_backward(x, dy, gamma, mean, variance, axes, eps, batch_stat, dmean, dvar, propagate_down, accum,
// grads): (dx, dbeta, dgamma), None where propagate_down is False
PyObject *batch_normalization_backward(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 13)
    return PyErr_Format(PyExc_TypeError, "expected 13 arguments, got %zd", nargs);
  Plain p;
  const at::Tensor *x = p.f32(a[0]), *dy = p.f32(a[1]), *gamma = p.f32_or_none(a[2]), *mean = p.f32(a[3]),
                   *var = p.f32(a[4]), *dmean = p.f32_or_none(a[8]), *dvar = p.f32_or_none(a[9]);
  const float eps = p.number(a[6]);
  const bool batch = p.truth(a[7]);
  bool down[3], accum[3];
  read_flags(p, a[10], down);
  read_flags(p, a[11], accum);
  p.require(axis_one(a[5]) && PyTuple_Check(a[12]) && PyTuple_GET_SIZE(a[12]) == 3 && p.ok && x->dim() >= 2 &&
            dy->sizes() == x->sizes());
  if (!p.ok)
    return not_plain();
  const int64_t outer = x->size(0), C = x->size(1), inner = x->numel() / std::max<int64_t>(outer * C, 1);
  for (const at::Tensor *t : {gamma, mean, var, dmean, dvar})
    p.require(!t || t->numel() == C);
  const at::IntArrayRef shapes[3] = {x->sizes(), at::IntArrayRef(C), at::IntArrayRef(C)};
  at::Tensor grad[3];
  for (int i = 0; p.ok && i < 3; ++i) {
    PyObject *given = PyTuple_GET_ITEM(a[12], i);
    if (!down[i])
      continue;
    if (given == Py_None) {
      p.require(!accum[i]);
    } else {
      const at::Tensor *t = p.f32(given);
      p.require(t && t->numel() == (i == 0 ? x->numel() : C));
      if (p.ok)
        grad[i] = *t;
    }
  }
  if (!p.ok)
    return not_plain();
  float *d[3] = {nullptr, nullptr, nullptr};
  for (int i = 0; i < 3; ++i)
    if (down[i]) {
      if (!grad[i].defined())
        grad[i] = empty_like_of(*x, shapes[i], at::kFloat);
      d[i] = data<float>(&grad[i]);
    }
  if (!run_on(*x, [&](void *stream) {
        return nb200_batch_normalization_backward_f32(data<float>(x), data<float>(dy), data<float>(gamma), data<float>(mean),
                                                      data<float>(var), data<float>(dmean), data<float>(dvar), d[0], d[1],
                                                      d[2], outer, C, inner, eps, batch, accum[0], accum[1], accum[2],
                                                      stream);
      }))
    return nullptr;
  PyObject *r = PyTuple_New(3);
  for (int i = 0; r && i < 3; ++i) {
    PyObject *given = PyTuple_GET_ITEM(a[12], i);
    PyObject *o = !down[i] ? Py_NewRef(Py_None) : given != Py_None ? Py_NewRef(given) : THPVariable_Wrap(grad[i]);
    PyTuple_SET_ITEM(r, i, o);
  }
  return r;
  END_HANDLE_TH_ERRORS
}

// The four ranges of a min-max quantizer: equal shapes of x's rank.
bool read_ranges(Plain &p, PyObject *const *a, const at::Tensor *x, const at::Tensor *(&q)[4]) {
  for (int i = 0; i < 4; ++i) {
    q[i] = p.f32(a[i]);
    p.require(p.ok && q[i]->dim() == x->dim() && q[i]->sizes() == q[0]->sizes());
  }
  return p.ok;
}

// min_max_quantize(x, qr_min, qr_max, ql_min, ql_max, decay, x_min_max, ema, eps): y
PyObject *min_max_quantize(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 9)
    return PyErr_Format(PyExc_TypeError, "expected 9 arguments, got %zd", nargs);
  Plain p;
  const at::Tensor *x = p.f32(a[0]), *q[4];
  const float decay = p.number(a[5]), eps = p.number(a[8]);
  const bool observe = p.truth(a[6]), ema = p.truth(a[7]);
  if (!p.ok || !read_ranges(p, a + 1, x, q))
    return not_plain();
  const at::Tensor y = empty_like_of(*x, x->sizes(), at::kFloat);
  if (!run_on(*x, [&](void *stream) {
        return nb200_min_max_quantize_f32(data<float>(x), x->sizes().data(), (int)x->dim(), data<float>(q[0]),
                                          data<float>(q[1]), data<float>(q[2]), data<float>(q[3]), q[0]->sizes().data(),
                                          decay, observe, ema, eps, data<float>(&y), nullptr, stream);
      }))
    return nullptr;
  return THPVariable_Wrap(y);
  END_HANDLE_TH_ERRORS
}

// min_max_quantize_backward(x, qr_min, qr_max, ql_min, ql_max, dy, x_min_max, ema, ste_fine_grained, propagate_down,
// accum, grads): (dx, g_qr_min, g_qr_max)
PyObject *min_max_quantize_backward(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 12)
    return PyErr_Format(PyExc_TypeError, "expected 12 arguments, got %zd", nargs);
  Plain p;
  const at::Tensor *x = p.f32(a[0]), *dy = p.f32(a[5]), *q[4];
  const bool observe = p.truth(a[6]), ema = p.truth(a[7]), fine = p.truth(a[8]);
  bool down[3], accum[3];
  read_flags(p, a[9], down);
  read_flags(p, a[10], accum);
  p.require(PyTuple_Check(a[11]) && PyTuple_GET_SIZE(a[11]) == 3);
  if (!p.ok || !read_ranges(p, a + 1, x, q))
    return not_plain();
  p.require(dy->sizes() == x->sizes());
  at::Tensor grad[3];
  for (int i = 0; p.ok && i < 3; ++i) {
    PyObject *given = PyTuple_GET_ITEM(a[11], i);
    if (given == Py_None) {
      p.require(!accum[i]);
    } else {
      const at::Tensor *t = p.f32(given);
      p.require(t && t->sizes() == (i == 0 ? x : q[0])->sizes());
      if (p.ok)
        grad[i] = *t;
    }
  }
  if (!p.ok)
    return not_plain();
  int32_t flags[3], add[3];
  for (int i = 0; i < 3; ++i) {
    flags[i] = down[i];
    add[i] = accum[i];
    if (!grad[i].defined()) {
      grad[i] = empty_like_of(*x, (i == 0 ? x : q[0])->sizes(), at::kFloat);
      flags[i] |= i == 0 ? 0 : 2; // a range gradient of this call's own: zero unless it is produced
    }
  }
  if (!run_on(*x, [&](void *stream) {
        return nb200_min_max_quantize_backward_f32(data<float>(x), x->sizes().data(), (int)x->dim(), data<float>(q[0]),
                                                   data<float>(q[1]), data<float>(q[2]), data<float>(q[3]),
                                                   q[0]->sizes().data(), data<float>(dy), observe, ema, fine, flags, add,
                                                   data<float>(&grad[0]), data<float>(&grad[1]), data<float>(&grad[2]),
                                                   stream);
      }))
    return nullptr;
  PyObject *r = PyTuple_New(3);
  for (int i = 0; r && i < 3; ++i) {
    PyObject *given = PyTuple_GET_ITEM(a[11], i);
    PyTuple_SET_ITEM(r, i, given != Py_None ? Py_NewRef(given) : THPVariable_Wrap(grad[i]));
  }
  return r;
  END_HANDLE_TH_ERRORS
}

#define ENTRY(name) {#name, (PyCFunction)(void (*)(void))Entry<name>::call, METH_FASTCALL, nullptr}
#define HELPER(name, fn) {name, (PyCFunction)(void (*)(void))fn, METH_FASTCALL, nullptr}

PyMethodDef methods[] = {
    ENTRY(nb200_fixed_point_quantize_f32),
    ENTRY(nb200_fixed_point_quantize_f32_codes),
    ENTRY(nb200_fixed_point_quantize_nhwc_codes_f32),
    ENTRY(nb200_fixed_point_quantize_backward_f32),
    ENTRY(nb200_pow2_quantize_f32),
    ENTRY(nb200_pow2_quantize_backward_f32),
    ENTRY(nb200_min_max_quantize_f32),
    ENTRY(nb200_min_max_quantize_backward_f32),
    ENTRY(nb200_binary_sigmoid_f32),
    ENTRY(nb200_binary_tanh_f32),
    ENTRY(nb200_binary_sigmoid_backward_f32),
    ENTRY(nb200_binary_tanh_backward_f32),
    ENTRY(nb200_quantize_linear_f32),
    ENTRY(nb200_dequantize_linear_f32),
    ENTRY(nb200_quantize_linear_backward_f32),
    ENTRY(nb200_dequantize_linear_backward_f32),
    ENTRY(nb200_prune_f32),
    ENTRY(nb200_prune_backward_f32),
    ENTRY(nb200_inq_restore_f32),
    ENTRY(nb200_inq_quantize_f32),
    ENTRY(nb200_affine_f32),
    ENTRY(nb200_affine_fxp8_f32),
    ENTRY(nb200_affine_codes_i8_f32),
    ENTRY(nb200_affine_codes_i8_kmajor_f32),
    ENTRY(nb200_transpose_codes_i8),
    ENTRY(nb200_affine_backward_f32),
    ENTRY(nb200_binary_weight_affine_f32),
    ENTRY(nb200_binary_connect_affine_f32),
    ENTRY(nb200_binary_weight_affine_backward_f32),
    ENTRY(nb200_binary_connect_affine_backward_f32),
    ENTRY(nb200_convolution_f32),
    ENTRY(nb200_convolution_fxp8_f32),
    ENTRY(nb200_convolution_backward_f32),
    ENTRY(nb200_convolution_input_backward_f32),
    ENTRY(nb200_convolution_codes_folded_nhwc),
    ENTRY(nb200_convolution_relu_fxp_codes_nhwc),
    ENTRY(nb200_binary_weight_convolution_f32),
    ENTRY(nb200_binary_connect_convolution_f32),
    ENTRY(nb200_binary_weight_convolution_backward_f32),
    ENTRY(nb200_binary_connect_convolution_backward_f32),
    ENTRY(nb200_binary_convolution_codes_f32),
    ENTRY(nb200_binary_convolution_codes_prepared_f32),
    ENTRY(nb200_binary_weights_prepare_i8),
    ENTRY(nb200_fixed_point_codes_nhwc),
    ENTRY(nb200_codes_nhwc_to_f32),
    ENTRY(nb200_global_average_pooling_codes_f32),
    ENTRY(nb200_max_pooling_f32),
    ENTRY(nb200_max_pooling_backward_f32),
    ENTRY(nb200_max_pooling_codes_nhwc),
    ENTRY(nb200_global_average_pooling_f32),
    ENTRY(nb200_global_average_pooling_backward_f32),
    ENTRY(nb200_batch_normalization_inference_f32),
    ENTRY(nb200_batch_normalization_batch_f32),
    ENTRY(nb200_batch_normalization_backward_f32),
    ENTRY(nb200_bn_add_relu_fxp_f32),
    ENTRY(nb200_bn_add_relu_fxp_codes_nhwc),
    ENTRY(nb200_relu_f32),
    ENTRY(nb200_relu_backward_f32),
    ENTRY(nb200_add2_f32),
    ENTRY(nb200_add2_backward_f32),
    {"calls", calls, METH_NOARGS, nullptr},
    HELPER("f32", f32),
    HELPER("empty", empty<at::kFloat>),
    HELPER("empty_i8", empty<at::kChar>),
    HELPER("conv2d", conv2d),
    HELPER("folded_convolution", folded_convolution),
    HELPER("folded_convolutions", folded_convolutions),
    HELPER("binary_convolution", binary_convolution),
    HELPER("binary_convolution_backward", binary_convolution_backward),
    HELPER("batch_normalization", batch_normalization),
    HELPER("min_max_quantize", min_max_quantize),
    HELPER("min_max_quantize_backward", min_max_quantize_backward),
    HELPER("batch_normalization_backward", batch_normalization_backward),
    HELPER("codes_nhwc_slots", codes_nhwc_slots),
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

} // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&module); }
