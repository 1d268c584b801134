// CPython entry points of the operators: the C-ABI functions of include/mace_b200.h that a program
// calls once per operator, callable from Python without ctypes.
//
// A small operator is over in three microseconds, and a ctypes call with two dozen arguments takes
// almost as long to convert them: the GPU then waits for the host between two launches (a 7 x 7
// depthwise convolution: one call per 6.4 us through ctypes, one per 2.6 us through this
// module).  The conversions are those of ctypes with declared argument types: integers are masked to the width of the
// parameter, None is a null pointer, anything with __float__ is a float.  The interpreter lock is
// released around the call, as ctypes does.
#include <Python.h>

#include <cstddef>
#include <tuple>
#include <type_traits>
#include <utility>

#include "../../include/mace_b200.h"

namespace {

template <typename T>
T Convert(PyObject *o) {
  if constexpr (std::is_pointer_v<T>) {
    return o == Py_None ? nullptr : reinterpret_cast<T>(PyLong_AsVoidPtr(o));
  } else if constexpr (std::is_floating_point_v<T>) {
    return static_cast<T>(PyFloat_AsDouble(o));
  } else {
    return static_cast<T>(PyLong_AsUnsignedLongLongMask(o));
  }
}

template <auto Fn, typename Sig>
struct Call;

template <auto Fn, typename... A>
struct Call<Fn, int (*)(A...)> {
  template <size_t... I>
  static PyObject *Run(PyObject *const *args, std::index_sequence<I...>) {
    std::tuple<A...> v{Convert<A>(args[I])...};
    if (PyErr_Occurred()) return nullptr;
    int status;
    Py_BEGIN_ALLOW_THREADS
    status = Fn(std::get<I>(v)...);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(status);
  }
  static PyObject *Entry(PyObject *, PyObject *const *args, Py_ssize_t n) {
    if (n != static_cast<Py_ssize_t>(sizeof...(A)))
      return PyErr_Format(PyExc_TypeError, "takes %zu arguments (%zd given)", sizeof...(A), n);
    return Run(args, std::index_sequence_for<A...>{});
  }
};

#define MB_ENTRY(name) \
  { #name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&Call<&name, decltype(&name)>::Entry)), METH_FASTCALL, nullptr }

PyMethodDef kMethods[] = {
    MB_ENTRY(mb_gemm_u8),
    MB_ENTRY(mb_gemv_u8),
    MB_ENTRY(mb_conv2d_u8_nhwc),
    MB_ENTRY(mb_dwconv_u8_nhwc),
    MB_ENTRY(mb_dwconv_u8_nhwc_prepacked),
    MB_ENTRY(mb_avgpool_u8_nhwc),
    MB_ENTRY(mb_gemm_f32),
    MB_ENTRY(mb_gemv_f32),
    MB_ENTRY(mb_conv2d_f32_nchw),
    MB_ENTRY(mb_conv2d_f32_nchw_residual),
    MB_ENTRY(mb_dwconv_f32_nchw),
    MB_ENTRY(mb_conv3x3_winograd_f32_nchw),
    MB_ENTRY(mb_pooling_f32_nchw),
    MB_ENTRY(mb_eltwise_act_f32),
    MB_ENTRY(mb_activation_f32),
    MB_ENTRY(mb_softmax_f32),
    MB_ENTRY(mb_quantize_f32_u8),
    MB_ENTRY(mb_dequantize_f32),
    MB_ENTRY(mb_transpose2d_batched),
    MB_ENTRY(mb_subsample_f32_nchw),
    MB_ENTRY(mb_stream_sync),
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_pycall", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__pycall() { return PyModule_Create(&kModule); }
