// CPython module `_pimb200_ops`: the call path of the short ops of `pimaicompiler_b200/ops.py` in native code.
//
// A batch-1 linear keeps the GPU busy for 3 us, but its checks, the output allocation and the foreign-function call took
// 8 us and more in Python, so a loop of such calls ran at the host's pace (4096 x 1024: 11.5 us per call).  Here a call
// is one C function: tensors are unpacked without a dispatcher, the output comes from the caching allocator directly,
// and the C ABI is called with the current stream.  Checks, messages and results are those of the Python functions.
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <vector>

#include "pimb200.h"

namespace {

struct PyError {};   // a Python exception has been set

[[noreturn]] void fail(PyObject* type, const char* msg) {
    PyErr_SetString(type, msg);
    throw PyError();
}

inline const at::Tensor& tensor(PyObject* o) {
    if (!THPVariable_Check(o)) fail(PyExc_TypeError, "expected a tensor");
    return THPVariable_Unpack(o);
}
inline void require_half_cuda(const at::Tensor& t) {
    if (!t.is_cuda() || t.scalar_type() != at::kHalf) fail(PyExc_TypeError, "expected a CUDA fp16 tensor");
}
inline const at::Tensor& half_contiguous(PyObject* o) {
    const at::Tensor& t = tensor(o);
    require_half_cuda(t);
    if (!t.is_contiguous()) fail(PyExc_ValueError, "expected a contiguous tensor");
    return t;
}
// (the address of a tensor without storage, such as a tracer's, is a C++ exception: asked for while Python's lock is held)
inline const void* half_or_null(PyObject* o) { return o == Py_None ? nullptr : half_contiguous(o).data_ptr(); }
inline void require(bool ok, const char* msg) {
    if (!ok) fail(PyExc_AssertionError, msg);
}
inline at::Tensor empty(at::IntArrayRef sizes, at::ScalarType dtype, const at::Tensor& like) {
    return at::Tensor(at::detail::empty_cuda(sizes, dtype, like.device(), std::nullopt));
}
inline void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
inline long as_long(PyObject* o) {
    const long v = PyLong_AsLong(o);
    if (v == -1 && PyErr_Occurred()) throw PyError();
    return v;
}
inline bool as_bool(PyObject* o) {
    const int v = PyObject_IsTrue(o);
    if (v < 0) throw PyError();
    return v != 0;
}

PyObject* g_check = nullptr;   // _lib.check(status, where): raises Pimb200Error

void check(int status, const char* where) {
    if (status == PIMB200_OK) return;
    PyObject* r = PyObject_CallFunction(g_check, "is", status, where);
    Py_XDECREF(r);
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, where);
    throw PyError();
}

// a call of the C ABI: other Python threads run meanwhile (it may allocate, or wait for another thread's call).  `call` takes
// addresses and numbers only
template <typename F>
int abi(F call) {
    struct Unlocked {
        PyThreadState* state = PyEval_SaveThread();
        ~Unlocked() { PyEval_RestoreThread(state); }
    } unlocked;
    return call();
}

// runs f and turns C++ exceptions into Python ones
template <typename F>
PyObject* guarded(F f) {
    try {
        return f();
    } catch (const PyError&) {
        return nullptr;
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

// the caller's `out` (returned itself) or a fresh tensor
struct Out {
    at::Tensor own;
    PyObject* given = nullptr;
    const at::Tensor& get() const { return given ? THPVariable_Unpack(given) : own; }
    PyObject* release() {
        if (given) {
            Py_INCREF(given);
            return given;
        }
        return THPVariable_Wrap(std::move(own));
    }
};
Out output(PyObject* given, at::IntArrayRef sizes, at::ScalarType dtype, const at::Tensor& like) {
    Out o;
    if (given != Py_None) {
        tensor(given);
        o.given = given;
    } else {
        o.own = empty(sizes, dtype, like);
    }
    return o;
}

// gemv_mv(W, x, bias, act, out)
PyObject* gemv_mv(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 5) fail(PyExc_TypeError, "gemv_mv takes 5 arguments");
        const at::Tensor &W = half_contiguous(a[0]), &x = half_contiguous(a[1]);
        const void* bias = half_or_null(a[2]);
        if (W.dim() != 2) fail(PyExc_ValueError, "expected a 2-D weight matrix");
        const int64_t N = W.size(0), K = W.size(1);
        require(x.numel() == K, "x does not have one element per column of W");
        const int act = (int)as_long(a[3]);
        Out y = output(a[4], {N}, at::kHalf, W);
        const void *wp = W.data_ptr(), *xp = x.data_ptr();
        void *yp = y.get().data_ptr(), *st = stream();
        check(abi([&] { return pimb200_gemv_mv(wp, xp, bias, yp, (int)N, (int)K, act, st); }), "gemv_mv");
        return y.release();
    });
}

// gemv_vm(x, A, bias, act, out)
PyObject* gemv_vm(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 5) fail(PyExc_TypeError, "gemv_vm takes 5 arguments");
        const at::Tensor &x = half_contiguous(a[0]), &A = half_contiguous(a[1]);
        const void* bias = half_or_null(a[2]);
        if (A.dim() != 2) fail(PyExc_ValueError, "expected a 2-D weight matrix");
        const int64_t K = A.size(0), N = A.size(1);
        require(x.numel() == K, "x does not have one element per row of A");
        const int act = (int)as_long(a[3]);
        Out y = output(a[4], {N}, at::kHalf, A);
        const void *xp = x.data_ptr(), *ap = A.data_ptr();
        void *yp = y.get().data_ptr(), *st = stream();
        check(abi([&] { return pimb200_gemv_vm(xp, ap, bias, yp, (int)K, (int)N, act, st); }), "gemv_vm");
        return y.release();
    });
}

// gemm_wx(W, X, bias, act, out_f32, out): rows of X and of out may be strided.  FIXED: gemm_wx_fixed
template <bool FIXED>
PyObject* gemm_wx(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 6) fail(PyExc_TypeError, "gemm_wx takes 6 arguments");
        const at::Tensor& W = half_contiguous(a[0]);
        const void* bias = half_or_null(a[2]);
        const at::Tensor& X = tensor(a[1]);
        require_half_cuda(X);
        if (X.dim() && X.stride(-1) != 1) fail(PyExc_ValueError, "expected a contiguous last dimension");
        if (W.dim() != 2) fail(PyExc_ValueError, "expected a 2-D weight matrix");
        const int64_t N = W.size(0), K = W.size(1);
        require(X.dim() >= 2 && X.size(1) == K && X.stride(1) == 1, "X does not have the columns of W");
        const int64_t J = X.size(0);
        const int act = (int)as_long(a[3]);
        Out y = output(a[5], {J, N}, as_bool(a[4]) ? at::kFloat : at::kHalf, W);
        const at::Tensor& Y = y.get();
        const void *wp = W.data_ptr(), *xp = X.data_ptr();
        void *yp = Y.data_ptr(), *st = stream();
        const int ldx = (int)X.stride(0), ldy = (int)Y.stride(0), f32 = Y.scalar_type() == at::kFloat ? 1 : 0;
        check(abi([&] { return (FIXED ? pimb200_gemm_wx_fixed : pimb200_gemm_wx)(wp, xp, bias, yp, (int)N, (int)K, (int)J, ldx, ldy, act, f32, st); }), "gemm_wx");
        return y.release();
    });
}

// The three outputs of an LSTM call: the caller's tuple (None = not wanted), or fresh tensors
struct LstmOut {
    Out y, hn, cn;
    PyObject* release() {
        PyObject* t = PyTuple_New(3);
        if (!t) throw PyError();
        PyTuple_SET_ITEM(t, 0, y.release());
        PyTuple_SET_ITEM(t, 1, hn.release());
        PyTuple_SET_ITEM(t, 2, cn.release());
        return t;
    }
};

// lstm_forward(handle, layers * directions, directions, hidden, x, h0, c0, batch_first, out): out is None or a tuple (y, hn, cn)
PyObject* lstm_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 9) fail(PyExc_TypeError, "lstm_forward takes 9 arguments");
        pimb200_lstm* h = static_cast<pimb200_lstm*>(PyLong_AsVoidPtr(a[0]));
        if (PyErr_Occurred()) throw PyError();
        const int64_t LD = as_long(a[1]), D = as_long(a[2]), H = as_long(a[3]);
        const at::Tensor& x = half_contiguous(a[4]);
        const void *h0 = half_or_null(a[5]), *c0 = half_or_null(a[6]);
        const bool bf = as_bool(a[7]);
        if (x.dim() != 3) fail(PyExc_ValueError, "expected a 3-D input");
        const int64_t B = x.size(bf ? 0 : 1), T = x.size(bf ? 1 : 0);
        if (a[8] != Py_None) {
            if (!PyTuple_Check(a[8]) || PyTuple_GET_SIZE(a[8]) != 3) fail(PyExc_ValueError, "out holds y, hn and cn");
            void* p[3];
            for (int i = 0; i < 3; ++i) {
                PyObject* t = PyTuple_GET_ITEM(a[8], i);
                p[i] = t == Py_None ? nullptr : tensor(t).data_ptr();
            }
            const void* xp = x.data_ptr();
            void* st = stream();
            check(abi([&] { return pimb200_lstm_forward(h, xp, (int)T, (int)B, h0, c0, p[0], p[1], p[2], bf ? 1 : 0, st); }), "lstm_forward");
            Py_INCREF(a[8]);
            return a[8];
        }
        LstmOut o;
        o.y.own = empty({x.size(0), x.size(1), D * H}, at::kHalf, x);
        o.hn.own = empty({LD, B, H}, at::kHalf, x);
        o.cn.own = empty({LD, B, H}, at::kHalf, x);
        const void* xp = x.data_ptr();
        void *yp = o.y.own.data_ptr(), *hp = o.hn.own.data_ptr(), *cp = o.cn.own.data_ptr(), *st = stream();
        check(abi([&] { return pimb200_lstm_forward(h, xp, (int)T, (int)B, h0, c0, yp, hp, cp, bf ? 1 : 0, st); }), "lstm_forward");
        return o.release();
    });
}

// lstm_forward_packed(handle, layers * directions, directions, hidden, data, batch_sizes, h0, c0)
PyObject* lstm_forward_packed(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 8) fail(PyExc_TypeError, "lstm_forward_packed takes 8 arguments");
        pimb200_lstm* h = static_cast<pimb200_lstm*>(PyLong_AsVoidPtr(a[0]));
        if (PyErr_Occurred()) throw PyError();
        const int64_t LD = as_long(a[1]), D = as_long(a[2]), H = as_long(a[3]);
        const at::Tensor& x = half_contiguous(a[4]);
        at::Tensor sizes = tensor(a[5]).to(at::kCPU, at::kLong).contiguous();
        if (sizes.dim() != 1 || sizes.numel() < 1) fail(PyExc_ValueError, "batch_sizes holds one whole number per step");
        const int64_t B = sizes.data_ptr<int64_t>()[0];
        const void *h0 = half_or_null(a[6]), *c0 = half_or_null(a[7]);
        LstmOut o;
        o.y.own = empty({x.size(0), D * H}, at::kHalf, x);
        o.hn.own = empty({LD, B, H}, at::kHalf, x);
        o.cn.own = empty({LD, B, H}, at::kHalf, x);
        const void* xp = x.data_ptr();
        const int64_t* sp = sizes.data_ptr<int64_t>();
        const int steps = (int)sizes.numel();
        void *yp = o.y.own.data_ptr(), *hp = o.hn.own.data_ptr(), *cp = o.cn.own.data_ptr(), *st = stream();
        check(abi([&] { return pimb200_lstm_forward_packed(h, xp, sp, steps, h0, c0, yp, hp, cp, st); }), "lstm_forward_packed");
        return o.release();
    });
}

PyObject* set_check(PyObject*, PyObject* f) {
    Py_INCREF(f);
    Py_XSETREF(g_check, f);
    Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"gemv_mv", (PyCFunction)(void (*)(void))gemv_mv, METH_FASTCALL, nullptr},
    {"gemv_vm", (PyCFunction)(void (*)(void))gemv_vm, METH_FASTCALL, nullptr},
    {"gemm_wx", (PyCFunction)(void (*)(void))gemm_wx<false>, METH_FASTCALL, nullptr},
    {"gemm_wx_fixed", (PyCFunction)(void (*)(void))gemm_wx<true>, METH_FASTCALL, nullptr},
    {"lstm_forward", (PyCFunction)(void (*)(void))lstm_forward, METH_FASTCALL, nullptr},
    {"lstm_forward_packed", (PyCFunction)(void (*)(void))lstm_forward_packed, METH_FASTCALL, nullptr},
    {"set_check", set_check, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_pimb200_ops", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__pimb200_ops() { return PyModule_Create(&kModule); }
