// The hot entry points of linear.py as a CPython extension: arguments in, one call of the C ABI, results out. A block is
// fifteen calls, and through ctypes each of them cost 10 to 12 us of host time beside the launch itself (two tensor
// allocations and a stream lookup through the Python bindings, seventeen converted arguments), more than most of the kernels
// of a small block run for: two prompts' cross-attention K and V took 40 us for 25 us of kernels. Here the same steps take
// about 3 us. linear.py keeps the signatures; what is not on a block's path stays on ctypes there.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "gpu_kernels.h"

namespace {

struct Error {};               // a Python exception is set

[[noreturn]] void raise(PyObject* type, const char* text) {
    PyErr_SetString(type, text);
    throw Error();
}
// The module's attribute `ok` (ffi.ok, put there by linear.py) raises the error a return code stands for.
[[noreturn]] void failed(PyObject* self, int rc, const char* what) {
    PyObject* r = PyObject_CallMethod(self, "ok", "is", rc, what);
    Py_XDECREF(r);
    if (r) PyErr_SetString(PyExc_RuntimeError, what);
    throw Error();
}
// One call of the C ABI without the interpreter lock (a launch can block on a full queue), as ctypes makes it.
template <typename... P, typename... A> void call(PyObject* self, const char* name, int (*f)(P...), A... args) {
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = f(static_cast<P>(args)...);
    Py_END_ALLOW_THREADS
    if (rc != 0) failed(self, rc, name);
}
#define CALL(f, ...) call(self, #f, f, __VA_ARGS__)
const at::Tensor* opt(PyObject* o) {
    if (o == Py_None) return nullptr;
    if (!THPVariable_Check(o)) raise(PyExc_TypeError, "expected a torch tensor");
    return &THPVariable_Unpack(o);
}
const at::Tensor& ten(PyObject* o) {
    const at::Tensor* t = opt(o);
    if (!t) raise(PyExc_TypeError, "expected a torch tensor");
    return *t;
}
const at::Tensor& on_gpu(PyObject* o) {
    const at::Tensor& t = ten(o);
    if (!t.is_cuda()) raise(PyExc_ValueError, "this path runs on CUDA tensors only");
    return t;
}
template <typename T = void> T* ptr(const at::Tensor* t) { return t ? reinterpret_cast<T*>(t->data_ptr()) : nullptr; }
template <typename T = void> T* ptr(const at::Tensor& t) { return reinterpret_cast<T*>(t.data_ptr()); }
int64_t integer(PyObject* o) {
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw Error();
    return v;
}
int integer32(PyObject* o) { return (int)integer(o); }
float real(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw Error();
    return (float)v;
}
int dtype_code(const at::Tensor& t) {
    switch (t.scalar_type()) {
        case at::kFloat: return 0;
        case at::kHalf: return 1;
        case at::kBFloat16: return 2;
        default: raise(PyExc_KeyError, c10::toString(t.scalar_type()));
    }
}
at::ScalarType out_dtype(PyObject* o) {
    if (!THPDtype_Check(o)) raise(PyExc_TypeError, "out_dtype is not a torch dtype");
    return reinterpret_cast<THPDtype*>(o)->scalar_type;
}
void rows_cols(const at::Tensor& t, int64_t& M, int64_t& K) {
    if (t.dim() != 2) raise(PyExc_ValueError, "expected a matrix");
    M = t.size(0), K = t.size(1);
}
at::Tensor matrix(const at::Tensor& like, int64_t M, int64_t K, at::ScalarType dt) {
    return at::empty({M, K}, at::TensorOptions().dtype(dt).device(like.device()));
}
at::Tensor vec(const at::Tensor& like, int64_t M, at::ScalarType dt = at::kFloat) {
    return at::empty({M}, at::TensorOptions().dtype(dt).device(like.device()));
}
at::Tensor given_or(PyObject* o, at::Tensor (*make)(const at::Tensor&, int64_t, int64_t, at::ScalarType), const at::Tensor& like, int64_t M,
                    int64_t K, at::ScalarType dt) {
    const at::Tensor* t = opt(o);
    return t ? *t : make(like, M, K, dt);
}
void* stream() { return (void*)c10::cuda::getCurrentCUDAStream().stream(); }
PyObject* wrap(PyObject* given, const at::Tensor& t) {
    if (given && given != Py_None) return Py_NewRef(given);
    return THPVariable_Wrap(t);
}
PyObject* pair(PyObject* ga, const at::Tensor& a, PyObject* gb, const at::Tensor& b) {
    PyObject* pa = wrap(ga, a);
    PyObject* pb = pa ? wrap(gb, b) : nullptr;
    PyObject* r = pb ? PyTuple_Pack(2, pa, pb) : nullptr;
    Py_XDECREF(pa), Py_XDECREF(pb);
    return r;
}
template <typename F> PyObject* guarded(Py_ssize_t have, Py_ssize_t want, F&& f) {
    HANDLE_TH_ERRORS                       // torch's own errors (out of memory among them) as its bindings raise them
    if (have != want) {
        PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, have);
        return nullptr;
    }
    try {
        return f();
    } catch (const Error&) {
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
}
#define FAST(name, n) PyObject* name(PyObject* self, PyObject* const* a, Py_ssize_t nargs) { return guarded(nargs, n, [&]() -> PyObject* {
#define END }); }

// x, prologue, rotate, K, g, up_offset, q, scales, norm_w, norm_b, eps, mod_scale, mod_shift
FAST(quant_rows, 13)
    const at::Tensor& x = on_gpu(a[0]);
    const int64_t M = x.size(0), K = a[3] == Py_None ? x.size(1) : integer(a[3]);
    at::Tensor q = given_or(a[6], matrix, x, M, K, at::kChar);
    const at::Tensor* given_s = opt(a[7]);
    at::Tensor s = given_s ? *given_s : vec(x, M);
    const at::Tensor *g = opt(a[4]), *nb = opt(a[9]);
    const int dt = dtype_code(x);
    if (nb)
        CALL(gpu_quant_rows_b, dt, integer32(a[1]), ptr(x), x.stride(0), ptr<float>(opt(a[8])), ptr<float>(nb), real(a[10]), ptr(opt(a[11])),
                               ptr(opt(a[12])), ptr<int8_t>(q), ptr<float>(s), (int)M, (int)K, integer32(a[2]), stream());
    else
        CALL(gpu_quant_rows, dt, integer32(a[1]), ptr(x), x.stride(0), ptr(g), g ? g->stride(0) : 0, integer(a[5]), ptr<float>(opt(a[8])), real(a[10]),
                             ptr(opt(a[11])), ptr(opt(a[12])), ptr<int8_t>(q), ptr<float>(s), (int)M, (int)K, integer32(a[2]), stream());
    return pair(a[6], q, a[7], s);
END
// x, rotate
FAST(sd_quant_rows, 2)
    const at::Tensor& x = on_gpu(a[0]);
    int64_t M, K;
    rows_cols(x, M, K);
    at::Tensor q = matrix(x, M, K, at::kChar), s = vec(x, M);
    CALL(gpu_sd_quant_rows, ptr(x), x.stride(0), ptr<int8_t>(q), ptr<float>(s), (int)M, (int)K, integer32(a[1]), stream());
    return pair(nullptr, q, nullptr, s);
END
// x, w, b, eps, rotate
FAST(sd_ln_quant_rows, 5)
    const at::Tensor& x = on_gpu(a[0]);
    int64_t M, K;
    rows_cols(x, M, K);
    at::Tensor q = matrix(x, M, K, at::kChar), s = vec(x, M);
    CALL(gpu_sd_ln_quant_rows, ptr(x), x.stride(0), ptr<float>(opt(a[1])), ptr<float>(opt(a[2])), real(a[3]), ptr<int8_t>(q), ptr<float>(s), (int)M, (int)K,
                               integer32(a[4]), stream());
    return pair(nullptr, q, nullptr, s);
END
// x, rotate
FAST(sd_geglu_quant_rows, 2)
    const at::Tensor& x = on_gpu(a[0]);
    const int64_t M = x.size(0), I = x.size(1) / 2;
    at::Tensor q = matrix(x, M, I, at::kChar), s = vec(x, M);
    CALL(gpu_sd_geglu_quant_rows, ptr(x), ptr<int8_t>(q), ptr<float>(s), (int)M, (int)I, integer32(a[1]), stream());
    return pair(nullptr, q, nullptr, s);
END
// x, w, b, groups, eps, rotate
FAST(sd_group_norm_quant_rows, 6)
    const at::Tensor& x = on_gpu(a[0]);
    if (x.dim() != 3) raise(PyExc_ValueError, "expected [N, P, C]");
    const int64_t N = x.size(0), P = x.size(1), C = x.size(2), G = integer(a[3]);
    at::Tensor q = matrix(x, N * P, C, at::kChar), s = vec(x, N * P), sums = vec(x, N * G * 2 + 2, at::kDouble);
    CALL(gpu_sd_group_norm_quant_rows, ptr(x), ptr<float>(opt(a[1])), ptr<float>(opt(a[2])), ptr(sums), (int)N, P, (int)C, (int)G, real(a[4]),
                                       ptr<int8_t>(q), ptr<float>(s), integer32(a[5]), stream());
    return pair(nullptr, q, nullptr, s);
END
// x, d, rotate
FAST(sd_unpad_quant_rows, 3)
    const at::Tensor& x = on_gpu(a[0]);
    if (x.dim() != 3) raise(PyExc_ValueError, "expected [M, H, dp]");
    const int64_t M = x.size(0), H = x.size(1), dp = x.size(2), d = integer(a[1]);
    at::Tensor q = matrix(x, M, H * d, at::kChar), s = vec(x, M);
    CALL(gpu_sd_unpad_quant_rows, ptr(x), ptr<int8_t>(q), ptr<float>(s), (int)M, (int)H, (int)d, (int)dp, integer32(a[2]), stream());
    return pair(nullptr, q, nullptr, s);
END
// A, W, xs, ws, bias, out_dtype, act, rscale, resid, out
FAST(int8_gemm, 10)
    const at::Tensor &A = on_gpu(a[0]), &W = ten(a[1]);
    int64_t M, K;
    rows_cols(A, M, K);
    const int64_t N = W.size(0);
    at::Tensor D = given_or(a[9], matrix, A, M, N, a[9] == Py_None ? out_dtype(a[5]) : at::kFloat);
    const int dt = dtype_code(D), act = integer32(a[6]);
    const at::Tensor *bias = opt(a[4]), *resid = opt(a[8]);
    const int8_t *pa = ptr<int8_t>(A), *pw = ptr<int8_t>(W);
    const float *xs = ptr<float>(opt(a[2])), *ws = ptr<float>(opt(a[3]));
    if (resid)
        CALL(gpu_int8_gemm_residual, pa, pw, xs, ws, ptr(bias), ptr(opt(a[7])), ptr(resid), ptr(D), M, N, K, dt, stream());
    else if (act) CALL(gpu_int8_gemm_act, pa, pw, xs, ws, ptr(bias), ptr(D), M, N, K, dt, act, stream());
    else CALL(gpu_int8_gemm, pa, pw, xs, ws, ptr(bias), ptr(D), M, N, K, dt, stream());
    return wrap(a[9], D);
END
// A, W, xs, ws, bias, act, out, amax_part
FAST(int8_gemm_act_rot, 8)
    const at::Tensor &A = on_gpu(a[0]), &W = ten(a[1]);
    int64_t M, K;
    rows_cols(A, M, K);
    const int64_t N = W.size(0);
    at::Tensor D = given_or(a[6], matrix, A, M, N, at::kBFloat16), parts = given_or(a[7], matrix, A, N / 64, M, at::kFloat);
    CALL(gpu_int8_gemm_act_rot, ptr<int8_t>(A), ptr<int8_t>(W), ptr<float>(opt(a[2])), ptr<float>(opt(a[3])), ptr(opt(a[4])), ptr(D), ptr<float>(parts),
                                M, N, K, integer32(a[5]), stream());
    return pair(a[6], D, a[7], parts);
END
// xr, amax_part, q, scales
FAST(quant_rows_rotated, 4)
    const at::Tensor& x = on_gpu(a[0]);
    int64_t M, K;
    rows_cols(x, M, K);
    at::Tensor q = given_or(a[2], matrix, x, M, K, at::kChar);
    const at::Tensor* given_s = opt(a[3]);
    at::Tensor s = given_s ? *given_s : vec(x, M);
    CALL(gpu_quant_rows_rotated, ptr(x), ptr<float>(ten(a[1])), ptr<int8_t>(q), ptr<float>(s), (int)M, (int)K, stream());
    return pair(a[2], q, a[3], s);
END
// A, packed, s_rel, xs, s_channel, bias, out_dtype, act, rscale, resid, out, G
FAST(w6a8_gemm, 12)
    const at::Tensor &A = on_gpu(a[0]), &W = ten(a[1]);
    int64_t M, K;
    rows_cols(A, M, K);
    const int64_t N = W.size(0);
    at::Tensor D = given_or(a[10], matrix, A, M, N, a[10] == Py_None ? out_dtype(a[6]) : at::kFloat);
    const int dt = dtype_code(D), act = integer32(a[7]), G = integer32(a[11]);
    const at::Tensor *bias = opt(a[5]), *resid = opt(a[9]);
    const int8_t* pa = ptr<int8_t>(A);
    const uint8_t *pw = ptr<uint8_t>(W), *rel = ptr<uint8_t>(opt(a[2]));
    const float *xs = ptr<float>(opt(a[3])), *ch = ptr<float>(opt(a[4]));
    if (resid)
        CALL(gpu_w6a8_gemm_residual, pa, pw, rel, xs, ch, ptr(bias), ptr(opt(a[8])), ptr(resid), ptr(D), M, N, K, G, dt, stream());
    else if (act) CALL(gpu_w6a8_gemm_act, pa, pw, rel, xs, ch, ptr(bias), ptr(D), M, N, K, G, dt, act, stream());
    else CALL(gpu_w6a8_gemm, pa, pw, rel, xs, ch, ptr(bias), ptr(D), M, N, K, G, dt, stream());
    return wrap(a[10], D);
END

#define M(name) {#name, (PyCFunction)(void (*)())name, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {M(quant_rows), M(sd_quant_rows), M(sd_ln_quant_rows), M(sd_geglu_quant_rows), M(sd_group_norm_quant_rows),
                         M(sd_unpad_quant_rows), M(int8_gemm), M(int8_gemm_act_rot), M(quant_rows_rotated), M(w6a8_gemm),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host_ops", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host_ops() { return PyModule_Create(&module); }
