// The Python call of the smallest operator without the interpreter's part: Context.linear through ctypes cost 8.9 us per call, of which
// 2.5 went into torch.empty, 2 into attribute reads and checks and 1 into converting eleven arguments, for a kernel of 3 us.  This
// module unpacks the tensors, allocates the result and calls mcu_linear (whose address it is given: the library stays the one
// that the package loaded).  Anything out of the ordinary is left to the Python code: FALLBACK.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/version.h>

typedef int (*LinearFn)(void *, int, const float *, size_t, const void *, size_t, size_t, size_t, const float *, float *, size_t);
static LinearFn g_linear = nullptr;
constexpr long FALLBACK = 1;  // (error codes of the library are negative)

static PyObject *set_entry_points(PyObject *, PyObject *arg) {
    g_linear = (LinearFn)PyLong_AsVoidPtr(arg);
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
}

// linear(context, kind, block values, block bytes, x, w, F, bias, out) -> the result, a negative error code, or FALLBACK
static PyObject *linear(PyObject *, PyObject *const *a, Py_ssize_t n) {
    HANDLE_TH_ERRORS  // (out of memory stays torch.OutOfMemoryError)
    if (n != 9 || g_linear == nullptr || !PyLong_CheckExact(a[0]) || !PyLong_CheckExact(a[1]) || !PyLong_CheckExact(a[2]) ||
        !PyLong_CheckExact(a[3]) || !THPVariable_Check(a[4]) || !THPVariable_Check(a[5]) || !PyLong_CheckExact(a[6]) ||
        (a[7] != Py_None && !THPVariable_Check(a[7])) || (a[8] != Py_None && !THPVariable_Check(a[8])))
        return PyLong_FromLong(FALLBACK);
    void *ctx = PyLong_AsVoidPtr(a[0]);
    const long kind = PyLong_AsLong(a[1]), values = PyLong_AsLong(a[2]), bytes = PyLong_AsLong(a[3]);
    const long long F = PyLong_AsLongLong(a[6]);
    if (PyErr_Occurred()) {
        PyErr_Clear();
        return PyLong_FromLong(FALLBACK);
    }
    const at::Tensor &x = THPVariable_Unpack(a[4]), &w = THPVariable_Unpack(a[5]);
    constexpr int64_t MOST = (int64_t)1 << 30;  // of a dimension (validate_linear in abi.cu): the products below do not overflow
    if (values <= 0 || F < 0 || F > MOST || x.dim() != 2 || !x.is_cuda() || !w.is_cuda() || x.stride(1) != 1) return PyLong_FromLong(FALLBACK);
    const int64_t T = x.size(0), K = x.size(1);
    if (K > MOST || w.numel() * (int64_t)w.element_size() < F * ((K + values - 1) / values * bytes)) return PyLong_FromLong(FALLBACK);
    at::Tensor made;
    const bool make = a[8] == Py_None;
    if (make) made = at::empty({T, F}, x.options().dtype(at::kFloat));
    const at::Tensor &out = make ? made : THPVariable_Unpack(a[8]);
    if (!make && out.dim() != 2) return PyLong_FromLong(FALLBACK);
    const float *bias = a[7] == Py_None ? nullptr : (const float *)THPVariable_Unpack(a[7]).data_ptr();
    const float *xp = (const float *)x.data_ptr();
    float *op = (float *)out.data_ptr();
    const void *wp = w.data_ptr();
    const size_t ldx = (size_t)x.stride(0), ldo = (size_t)out.stride(0);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = g_linear(ctx, (int)kind, xp, ldx, wp, (size_t)T, (size_t)K, (size_t)F, bias, op, ldo);
    Py_END_ALLOW_THREADS
    if (rc != 0) return PyLong_FromLong(rc);
    if (make) return THPVariable_Wrap(made);
    Py_INCREF(a[8]);
    return a[8];
    END_HANDLE_TH_ERRORS
}

static PyMethodDef methods[] = {
    {"set_entry_points", set_entry_points, METH_O, "address of mcu_linear"},
    {"linear", (PyCFunction)(void (*)(void))linear, METH_FASTCALL, "Context.linear"},
    {nullptr, nullptr, 0, nullptr},
};
static PyModuleDef module = {PyModuleDef_HEAD_INIT, "_binding", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};
PyMODINIT_FUNC PyInit__binding() {
    PyObject *m = PyModule_Create(&module);
    if (m != nullptr) PyModule_AddStringConstant(m, "torch_version", TORCH_VERSION);  // it is of no use to another one
    return m;
}
