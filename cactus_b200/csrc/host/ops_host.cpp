// The host path of the single-op entry points (cactus_b200/ops.py) in native code: argument checks, result and scratch
// allocation from torch's caching allocator, current stream, and the call into libcactus_b200.so.
//
// A product of one token is 5 us of GPU work; through ctypes the call cost 17 us of interpreter time (a dozen attribute
// reads, two torch.empty, argument conversion), so the GPU waited for the host.  This does the same in about 1 us plus
// the launches.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../../include/cactus_b200.h"

// what this file was compiled against: build.py rebuilds it, and _lib.py refuses it, where that is not what runs
extern "C" __attribute__((used, visibility("default"))) const char b200_host_abi[] = "b200_host_abi{" B200_HOST_ABI "}";

namespace {

PyObject *g_error = nullptr;   // cactus_b200._lib.B200Error

// the failure of a check: a Python exception is set
struct Fail {};

void require(bool ok, const char *what) {
    if (ok) return;
    PyErr_SetString(PyExc_AssertionError, what);
    throw Fail{};
}
void check(int rc) {
    if (rc == 0) return;
    PyErr_Format(g_error, "cactus_b200 error %d: %s", rc, b200_last_error());
    throw Fail{};
}
const at::Tensor &tensor(PyObject *o, const char *what) {
    if (!THPVariable_Check(o)) {
        PyErr_Format(PyExc_TypeError, "%s must be a tensor", what);
        throw Fail{};
    }
    return THPVariable_Unpack(o);
}
const at::Tensor *maybe_tensor(PyObject *o, const char *what) { return o == Py_None ? nullptr : &tensor(o, what); }
void need_cuda(const at::Tensor *t) {
    if (!t || t->is_cuda()) return;
    PyErr_SetString(g_error, "cactus_b200 ops need CUDA tensors; there is no CPU path");
    throw Fail{};
}
long long integer(PyObject *o) {
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw Fail{};
    return v;
}
double real(PyObject *o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw Fail{};
    return v;
}
at::Tensor bytes_like(const at::Tensor &t, size_t n) { return at::empty({(int64_t) n}, t.options().dtype(at::kByte)); }

// the interpreter is free for other threads while a call into the library launches (the launch queue may be full)
struct NoGil {
    PyThreadState *state = PyEval_SaveThread();
    ~NoGil() { PyEval_RestoreThread(state); }
};

// What torch throws reaches the caller as the exception that torch itself would raise: an allocation that fails is a
// torch.OutOfMemoryError, which callers catch to free memory and try again.  (Out of line: torch's macros set up a warning
// handler, 0.1 us of a call that takes 1 us on the host.)
PyObject *translated(std::exception_ptr e) {
    HANDLE_TH_ERRORS
    std::rethrow_exception(e);
    END_HANDLE_TH_ERRORS
}
template <typename F>
PyObject *guarded(F f) {
    try {
        return f();
    } catch (const Fail &) {
        return nullptr;
    } catch (...) {
        return translated(std::current_exception());
    }
}

// mul_mat(wtype, K, M, w_data, x, variant, out | None, scratch | None) -> out
PyObject *mul_mat(PyObject *, PyObject *const *a, Py_ssize_t n) {
    return guarded([&]() -> PyObject * {
        require(n == 8, "mul_mat takes 8 arguments");
        const int wtype = (int) integer(a[0]);
        const int64_t K = integer(a[1]), M = integer(a[2]);
        const at::Tensor &w = tensor(a[3], "w"), &x = tensor(a[4], "x");
        need_cuda(&x);
        require(x.scalar_type() == at::kFloat && x.dim() == 2 && x.stride(1) == 1 && x.size(1) == K, "x must be f32 [N, K] with contiguous rows");
        const int64_t N = x.size(0);
        c10::cuda::OptionalCUDAGuard device(x.device());
        const at::Tensor *given = maybe_tensor(a[6], "out"), *scratch = maybe_tensor(a[7], "scratch");
        need_cuda(given);
        const at::Tensor out = given ? *given : at::empty({N, M}, x.options());
        const size_t need = b200_mul_mat_scratch_bytes(wtype, K, M, N);
        at::Tensor own;
        if (!scratch || (size_t) scratch->numel() < need) {
            own = bytes_like(x, need);
            scratch = &own;
        }
        const int variant = (int) integer(a[5]);
        const auto run = [&] {
            NoGil nogil;
            return b200_mul_mat_q(wtype, w.data_ptr(), K, M, (const float *) x.data_ptr(), x.stride(0) * 4, N, (float *) out.data_ptr(), out.stride(0) * 4,
                             scratch->data_ptr(), (size_t) scratch->numel(), variant, c10::cuda::getCurrentCUDAStream(x.device().index()).stream());
        };
        check(run());
        return THPVariable_Wrap(out);
    });
}

// flash_attn_ext(q, k, v, mask | None, scale, max_bias, logit_softcap, n_kv) -> out
PyObject *flash_attn_ext(PyObject *, PyObject *const *a, Py_ssize_t n) {
    return guarded([&]() -> PyObject * {
        require(n == 8, "flash_attn_ext takes 8 arguments");
        const at::Tensor &q = tensor(a[0], "q"), &k = tensor(a[1], "k"), &v = tensor(a[2], "v");
        const at::Tensor *mask = maybe_tensor(a[3], "mask");
        need_cuda(&q);
        need_cuda(&k);
        need_cuda(&v);
        need_cuda(mask);
        require(q.dim() == 3 && k.dim() == 3 && v.dim() == 3, "q [Nq, H, D], k and v [cells, Hkv, D]");
        require(q.scalar_type() == at::kFloat && k.scalar_type() == at::kHalf && v.scalar_type() == at::kHalf, "q must be f32, k and v f16");
        require(q.stride(2) == 1 && k.stride(2) == 1 && v.stride(2) == 1, "the head dimension must be contiguous");
        const int64_t Nq = q.size(0), H = q.size(1), D = q.size(2), Hkv = k.size(1), n_kv = integer(a[7]);
        if (mask) require(mask->scalar_type() == at::kHalf && mask->dim() == 2 && mask->stride(1) == 1 && mask->size(1) >= n_kv, "mask must be f16 [>= Nq, n_kv]");
        c10::cuda::OptionalCUDAGuard device(q.device());
        const at::Tensor out = at::empty({Nq, H, D}, q.options());
        const size_t need = b200_flash_attn_scratch_bytes(D, H, Hkv, Nq, n_kv);
        const at::Tensor scratch = bytes_like(q, need > 256 ? need : 256);
        const float scale = (float) real(a[4]), max_bias = (float) real(a[5]), softcap = (float) real(a[6]);
        const auto run = [&] {
            NoGil nogil;
            return b200_flash_attn_ext(D, H, Hkv, Nq, n_kv, (const float *) q.data_ptr(), q.stride(0) * 4, q.stride(1) * 4, k.data_ptr(), k.stride(0) * 2, k.stride(1) * 2,
                                  v.data_ptr(), v.stride(0) * 2, v.stride(1) * 2, mask ? mask->data_ptr() : nullptr, mask ? mask->stride(0) * 2 : 0,
                                  scale, max_bias, softcap, (float *) out.data_ptr(), scratch.data_ptr(), (size_t) scratch.numel(),
                                  c10::cuda::getCurrentCUDAStream(q.device().index()).stream());
        };
        check(run());
        return THPVariable_Wrap(out);
    });
}

PyMethodDef methods[] = {{"mul_mat", (PyCFunction) (void *) mul_mat, METH_FASTCALL, nullptr},
                         {"flash_attn_ext", (PyCFunction) (void *) flash_attn_ext, METH_FASTCALL, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_ops_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__ops_host(void) {
    PyObject *lib = PyImport_ImportModule("cactus_b200._lib");
    if (!lib) return nullptr;
    g_error = PyObject_GetAttrString(lib, "B200Error");
    Py_DECREF(lib);
    return g_error ? PyModule_Create(&module) : nullptr;
}
