// The flat C ABI as functions of a Python module: what cunn_b200/functional.py calls for every layer.
//
// A small layer is over on the GPU before its call is: through ctypes, which looks up a converter for each of 14 arguments, a call takes
// 5 us (2.4 us for a size with 11 integers), here 0.5.  The arguments' types come from include/cunn_b200.h; integers, numbers and addresses
// are taken and refused as ctypes does with those types: an int or what has an __index__ for an integer, an int or None for a pointer, what
// converts to float for a float, ctypes.ArgumentError otherwise.  What ctypes takes beside them, instances of its own types and, as pointers,
// bytes, is refused.  Like ctypes, a call runs without the interpreter's lock.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <tuple>
#include <type_traits>
#include <utility>

#include "../../../include/cunn_b200.h"

namespace {

PyObject *g_argument_error;

template <class T>
bool convert(PyObject *o, T &v)
{
    if constexpr (std::is_floating_point_v<T>) {
        const double d = PyFloat_AsDouble(o);
        v = (T)d;
        return d != -1.0 || !PyErr_Occurred();
    } else if constexpr (std::is_pointer_v<T>) {
        if (o == Py_None) {
            v = nullptr;
            return true;
        }
        if (!PyLong_Check(o)) return false;
        v = (T)(uintptr_t)PyLong_AsUnsignedLongLongMask(o);
        return true;
    } else {
        static_assert(std::is_integral_v<T>);
        v = (T)PyLong_AsUnsignedLongLongMask(o);               // by __index__, if it is not an int
        return v != (T)-1 || !PyErr_Occurred();
    }
}

template <class R, class... A, size_t... I>
PyObject *invoke(R (*f)(A...), PyObject *const *args, Py_ssize_t n, std::index_sequence<I...>)
{
    if (n != (Py_ssize_t)sizeof...(A)) {
        PyErr_Format(PyExc_TypeError, "this function takes %d arguments (%zd given)", (int)sizeof...(A), n);
        return nullptr;
    }
    std::tuple<std::remove_cv_t<A>...> v;
    int bad = -1;
    (void)((convert(args[I], std::get<I>(v)) || (bad = (int)I, false)) && ...);
    if (bad >= 0) {
        PyErr_Clear();
        PyErr_Format(g_argument_error, "argument %d: wrong type %s", bad + 1, Py_TYPE(args[bad])->tp_name);
        return nullptr;
    }
    R r;
    Py_BEGIN_ALLOW_THREADS
    r = f(std::get<I>(v)...);
    Py_END_ALLOW_THREADS
    if constexpr (std::is_same_v<R, size_t>) return PyLong_FromSize_t(r);
    else return PyLong_FromLong(r);
}
template <class R, class... A>
PyObject *invoke(R (*f)(A...), PyObject *const *args, Py_ssize_t n)
{
    return invoke(f, args, n, std::index_sequence_for<A...>());
}
template <auto F>
PyObject *call(PyObject *, PyObject *const *args, Py_ssize_t n)
{
    return invoke(F, args, n);
}

#define CALL(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&call<&name>)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {
    CALL(cunn_b200_adaptive_avgpool_backward),
    CALL(cunn_b200_adaptive_avgpool_forward),
    CALL(cunn_b200_adaptive_maxpool_backward),
    CALL(cunn_b200_adaptive_maxpool_forward),
    CALL(cunn_b200_avgpool_backward),
    CALL(cunn_b200_avgpool_forward),
    CALL(cunn_b200_batchnorm_backward),
    CALL(cunn_b200_batchnorm_forward),
    CALL(cunn_b200_batchnorm_relu_backward),
    CALL(cunn_b200_batchnorm_relu_forward),
    CALL(cunn_b200_batchnorm_workspace),
    CALL(cunn_b200_classnll_backward),
    CALL(cunn_b200_classnll_forward),
    CALL(cunn_b200_conv_forward_scratch),
    CALL(cunn_b200_conv_grad_input_scratch),
    CALL(cunn_b200_conv_scratch),
    CALL(cunn_b200_convmm_acc_grad),
    CALL(cunn_b200_convmm_acc_grad_workspace),
    CALL(cunn_b200_convmm_forward),
    CALL(cunn_b200_convmm_grad_input),
    CALL(cunn_b200_dilated_conv_acc_grad),
    CALL(cunn_b200_dilated_conv_acc_grad_workspace),
    CALL(cunn_b200_dwconv_acc_grad),
    CALL(cunn_b200_dwconv_acc_grad_workspace),
    CALL(cunn_b200_dwconv_forward),
    CALL(cunn_b200_dwconv_grad_input),
    CALL(cunn_b200_full_conv_acc_grad),
    CALL(cunn_b200_full_conv_acc_grad_workspace),
    CALL(cunn_b200_full_conv_forward_scratch),
    CALL(cunn_b200_full_conv_grad_input_scratch),
    CALL(cunn_b200_full_conv_scratch),
    CALL(cunn_b200_local_conv_acc_grad),
    CALL(cunn_b200_local_conv_forward),
    CALL(cunn_b200_local_conv_grad_input),
    CALL(cunn_b200_logsoftmax_backward),
    CALL(cunn_b200_logsoftmax_forward),
    CALL(cunn_b200_maxpool_backward),
    CALL(cunn_b200_maxpool_forward),
    CALL(cunn_b200_maxpool_out_size),
    CALL(cunn_b200_sgd_update),
    CALL(cunn_b200_threshold_backward),
    CALL(cunn_b200_threshold_forward),
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_calls", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__calls()
{
    PyObject *ctypes = PyImport_ImportModule("ctypes");
    if (!ctypes) return nullptr;
    g_argument_error = PyObject_GetAttrString(ctypes, "ArgumentError");
    Py_DECREF(ctypes);
    PyObject *m = g_argument_error ? PyModule_Create(&g_module) : nullptr;
    if (m && PyModule_AddIntConstant(m, "CONV_POINT_VALUES", CUNN_B200_CONV_POINT_VALUES)) Py_CLEAR(m);
    return m;
}
