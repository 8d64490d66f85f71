// Host side of the Python mirror: the C ABI's entry points as Python functions that take torch tensors.
//
// What bounds a small call is the host. Through ctypes an entry point with twenty arguments cost 4 to 6 us of
// argument objects before its kernel launch (2.1 us), and the shape arithmetic and allocations of the Python
// mirror as much again. Here each argument is read straight from its Python object by the parameter's C type, the
// device and stream come from the tensors, and the helpers below do the mirror's per-call checks and allocations.
// Measured per call, before and after, with the launch: ReLU of a small tensor 8.2 -> 4.7 us, a binary-weight
// convolution 21.8 -> 10.3 us, a folded convolution 23.4 -> 7.2 us; the folded ResNet-18 on one image 587 -> 235 us.
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <array>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <tuple>
#include <type_traits>
#include <utility>

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
    const int current = c10::cuda::current_device();
    if (device >= 0 && device != current)
      c10::cuda::set_device((c10::DeviceIndex)device);
    std::get<n>(a).v = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)(device >= 0 ? device : current)).stream();
    g_calls.fetch_add(1, std::memory_order_relaxed);
    int rc;
    Py_BEGIN_ALLOW_THREADS;
    rc = std::apply([](auto &...x) { return Fn(x.v...); }, a);
    Py_END_ALLOW_THREADS;
    if (device >= 0 && device != current)
      c10::cuda::set_device((c10::DeviceIndex)current);
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

// conv2d(x, w, bias, base_axis, pad, stride, dilation, group): the geometry of a 2-D convolution with one batch axis,
// (batch, channels, height, width, outmaps, kh, kw, pad, stride, dilation, output shape); x and w are tensors or
// shapes. None where the operands are of another form or do not fit together: the caller's full checks say why.
PyObject *conv2d(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 8)
    return PyErr_Format(PyExc_TypeError, "expected 8 arguments, got %zd", nargs);
  c10::SmallVector<int64_t, 8> x, w;
  int64_t pad[2], stride[2], dil[2], out[2];
  const long base_axis = PyLong_AsLong(args[3]), group = PyLong_AsLong(args[7]);
  bool ok = !PyErr_Occurred() && read_shape(args[0], x) && read_shape(args[1], w) && x.size() == 4 && w.size() == 4 &&
            base_axis == 1 && read_pair(args[4], 0, pad) && read_pair(args[5], 1, stride) &&
            read_pair(args[6], 1, dil) && group > 0 && x[1] % group == 0 && w[0] % group == 0 && x[1] / group == w[1];
  if (ok && args[2] != Py_None) {
    c10::SmallVector<int64_t, 8> b;
    ok = read_shape(args[2], b) && b.size() == 1 && b[0] == w[0];
  }
  for (int i = 0; ok && i < 2; ++i) {
    const int64_t span = x[2 + i] + 2 * pad[i] - (dil[i] * (w[2 + i] - 1) + 1);
    ok = span >= 0 && stride[i] > 0;
    out[i] = ok ? span / stride[i] + 1 : 0;
  }
  if (!ok) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  return Py_BuildValue("LLLLLLL(LL)(LL)(LL)(LLLL)", (long long)x[0], (long long)x[1], (long long)x[2], (long long)x[3],
                       (long long)w[0], (long long)w[2], (long long)w[3], (long long)pad[0], (long long)pad[1],
                       (long long)stride[0], (long long)stride[1], (long long)dil[0], (long long)dil[1],
                       (long long)x[0], (long long)w[0], (long long)out[0], (long long)out[1]);
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
    HELPER("codes_nhwc_slots", codes_nhwc_slots),
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

} // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&module); }
