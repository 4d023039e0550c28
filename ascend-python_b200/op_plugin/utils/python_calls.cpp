// Calls from Python to the operators that a decode step makes many of, without torch.ops' schema matching.
//
// torch.ops converts every argument to a boxed value, matches it against the schema and unboxes it again; for kernels of 2 to
// 5 us that took longer than the launch (one 1 x 1024 row: npu_dynamic_quant 6.8 us a call, of them 2.0 the C ABI with its
// launch).  A function here reads its arguments itself and calls the same operator through the dispatcher, so autograd,
// tracing, functorch and dispatch modes see what they saw before.  What it does not know - subclasses of Tensor, an active
// __torch_function__ mode, arguments of other types - it leaves to torch.ops: it returns NotImplemented.
//
// A Python extension module of its own (ops_loader.py): the operators are looked up by name in the dispatcher, so the library that
// registers them needs no Python and a C++ program can load it.
#include <torch/csrc/python_headers.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/dispatch/Dispatcher.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "op_plugin/utils/Export.h"

namespace {

using Optional = c10::optional<at::Tensor>;

// Reads positional arguments; `ok` turns false at the first one that torch.ops has to look at.
struct Arguments {
    PyObject *const *args;
    bool ok;
    Arguments(PyObject *const *a, Py_ssize_t given, Py_ssize_t wanted)
        : args(a), ok(given == wanted && !at::impl::torch_function_mode_enabled())
    {
    }
    const at::Tensor &tensor(int i)
    {
        static const at::Tensor none;
        ok = ok && THPVariable_CheckExact(args[i]);
        return ok ? THPVariable_Unpack(args[i]) : none;
    }
    Optional optional(int i) { return ok && args[i] == Py_None ? Optional() : Optional(tensor(i)); }
    int64_t integer(int i)
    {
        ok = ok && PyLong_CheckExact(args[i]);
        if (!ok) return 0;
        int overflow = 0;
        const long long v = PyLong_AsLongLongAndOverflow(args[i], &overflow);
        ok = overflow == 0;
        return v;
    }
    double number(int i)
    {
        ok = ok && PyFloat_CheckExact(args[i]);
        return ok ? PyFloat_AS_DOUBLE(args[i]) : 0.0;
    }
    c10::optional<at::ScalarType> dtype(int i)
    {
        if (!ok || args[i] == Py_None) return c10::nullopt;
        ok = THPDtype_Check(args[i]);
        if (!ok) return c10::nullopt;
        return reinterpret_cast<THPDtype *>(args[i])->scalar_type;
    }
};

PyObject *not_here()
{
    Py_RETURN_NOTIMPLEMENTED;
}

PyObject *wrap(at::Tensor &&t) { return THPVariable_Wrap(std::move(t)); }
template <typename... T>
PyObject *wrap(std::tuple<T...> &&t)
{
    PyObject *out = PyTuple_New(sizeof...(T));
    if (out == nullptr) throw python_error();
    Py_ssize_t i = 0;
    std::apply([&](auto &&...v) { (PyTuple_SET_ITEM(out, i++, THPVariable_Wrap(std::move(v))), ...); }, std::move(t));
    return out;
}

template <typename Op, typename... A>
PyObject *call(const Op &op, const A &...a)
{
    return wrap([&] {
        pybind11::gil_scoped_release release;
        return op.call(a...);
    }());
}

template <typename Signature>
c10::TypedOperatorHandle<Signature> find(const char *name)
{
    return c10::Dispatcher::singleton().findSchemaOrThrow(name, "").typed<Signature>();
}

PyObject *dynamic_quant(PyObject *, PyObject *const *args, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    static const auto op = find<std::tuple<at::Tensor, at::Tensor>(const at::Tensor &, const Optional &)>("npu::npu_dynamic_quant");
    Arguments a(args, n, 2);
    if (!a.ok) return not_here();
    const at::Tensor &x = a.tensor(0);
    const Optional smooth = a.optional(1);
    return a.ok ? call(op, x, smooth) : not_here();
    END_HANDLE_TH_ERRORS
}

PyObject *rms_norm(PyObject *, PyObject *const *args, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    static const auto op = find<std::tuple<at::Tensor, at::Tensor>(const at::Tensor &, const at::Tensor &, double)>("npu::npu_rms_norm");
    Arguments a(args, n, 3);
    if (!a.ok) return not_here();
    const at::Tensor &x = a.tensor(0), &gamma = a.tensor(1);
    const double eps = a.number(2);
    return a.ok ? call(op, x, gamma, eps) : not_here();
    END_HANDLE_TH_ERRORS
}

PyObject *rms_norm_dynamic_quant(PyObject *, PyObject *const *args, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    static const auto op = find<std::tuple<at::Tensor, at::Tensor, at::Tensor>(const at::Tensor &, const at::Tensor &, double)>(
        "npu::npu_rms_norm_dynamic_quant");
    Arguments a(args, n, 3);
    if (!a.ok) return not_here();
    const at::Tensor &x = a.tensor(0), &gamma = a.tensor(1);
    const double eps = a.number(2);
    return a.ok ? call(op, x, gamma, eps) : not_here();
    END_HANDLE_TH_ERRORS
}

PyObject *quant_matmul(PyObject *, PyObject *const *args, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    static const auto op = find<at::Tensor(const at::Tensor &, const at::Tensor &, const at::Tensor &, const Optional &,
                                           const Optional &, const Optional &, c10::optional<at::ScalarType>)>("npu::npu_quant_matmul");
    Arguments a(args, n, 7);
    if (!a.ok) return not_here();
    const at::Tensor &x1 = a.tensor(0), &x2 = a.tensor(1), &scale = a.tensor(2);
    const Optional offset = a.optional(3), pertoken = a.optional(4), bias = a.optional(5);
    const auto dtype = a.dtype(6);
    return a.ok ? call(op, x1, x2, scale, offset, pertoken, bias, dtype) : not_here();
    END_HANDLE_TH_ERRORS
}

PyObject *weight_quant_batchmatmul(PyObject *, PyObject *const *args, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    static const auto op = find<at::Tensor(const at::Tensor &, const at::Tensor &, const at::Tensor &, const Optional &,
                                           const Optional &, const Optional &, const Optional &, int64_t)>("npu::npu_weight_quant_batchmatmul");
    Arguments a(args, n, 8);
    if (!a.ok) return not_here();
    const at::Tensor &x = a.tensor(0), &weight = a.tensor(1), &scale = a.tensor(2);
    const Optional offset = a.optional(3), qscale = a.optional(4), qoffset = a.optional(5), bias = a.optional(6);
    const int64_t group = a.integer(7);
    return a.ok ? call(op, x, weight, scale, offset, qscale, qoffset, bias, group) : not_here();
    END_HANDLE_TH_ERRORS
}

template <PyObject *(*F)(PyObject *, PyObject *const *, Py_ssize_t)>
PyMethodDef method(const char *name)
{
    return {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(F)), METH_FASTCALL, nullptr};
}

PyMethodDef methods[] = {method<dynamic_quant>("dynamic_quant"),
                         method<rms_norm>("rms_norm"),
                         method<rms_norm_dynamic_quant>("rms_norm_dynamic_quant"),
                         method<quant_matmul>("quant_matmul"),
                         method<weight_quant_batchmatmul>("weight_quant_batchmatmul"),
                         {nullptr, nullptr, 0, nullptr}};

PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_op_plugin_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" OP_PLUGIN_EXPORT PyObject *PyInit__op_plugin_calls() { return PyModule_Create(&module_def); }
