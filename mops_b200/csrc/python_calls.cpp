// The functions of mops_b200 on CUDA tensors, called straight from the interpreter.
//
// `call(operation, arguments...)` does what the Python front end does for the ordinary case: plain
// contiguous CUDA tensors of one device, f32 or f64 throughout, int32 indices, the right numbers of
// dimensions. It allocates the results, points the library at torch's current stream, calls the C
// ABI with the interpreter lock released and returns the results. For anything else (host arrays,
// other index types, views, wrong arguments) it returns NotImplemented and the front end takes its
// general path, with its checks and messages. A call of the front end on 60 000 entries spends 40
// to 100 us in Python on its way to a 20 us kernel; this way it is a few.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/torch.h>

#include "../../include/mops.h"

namespace {

using at::Tensor;

PyObject* g_error = nullptr; // mops_b200.MopsError

// A tensor (or nullptr: a skipped gradient) as any of the ABI's by-value structs.
struct Arg {
    const Tensor* t;
    template <typename S> operator S() const {
        S s{};
        constexpr size_t n = sizeof(s.shape) / sizeof(s.shape[0]);
        if (t != nullptr && t->defined()) {
            s.data = static_cast<decltype(s.data + 0)>(t->data_ptr());
            for (size_t d = 0; d < n; d++) s.shape[d] = t->size(static_cast<int64_t>(d));
        }
        return s;
    }
};

// The arguments of one call, checked as they are taken.
struct Args {
    PyObject* const* args;
    Py_ssize_t n, at = 0;
    bool ok = true;
    const Tensor* first = nullptr;

    const Tensor* tensor(int64_t dims) {
        if (!ok || at >= n || !THPVariable_CheckExact(args[at])) return fail();
        const Tensor* t = &THPVariable_Unpack(args[at++]);
        if (!t->is_cuda() || t->layout() != at::kStrided || t->dim() != dims || !t->is_contiguous() ||
            t->is_neg() || t->is_conj())
            return fail();
        if (first == nullptr) first = t;
        if (t->device() != first->device()) return fail();
        return t;
    }
    const Tensor* real(int64_t dims) {
        const Tensor* t = tensor(dims);
        if (t == nullptr) return nullptr;
        const auto type = t->scalar_type();
        if ((type != at::kFloat && type != at::kDouble) || type != first->scalar_type()) return fail();
        return t;
    }
    const Tensor* index(int64_t dims) {
        const Tensor* t = tensor(dims);
        if (t != nullptr && t->scalar_type() != at::kInt) return fail();
        return t;
    }
    int64_t size() {
        if (!ok || at >= n || !PyLong_CheckExact(args[at])) {
            ok = false;
            return 0;
        }
        const int64_t v = PyLong_AsLongLong(args[at++]);
        if (v < 0) {
            PyErr_Clear();
            ok = false;
        }
        return v;
    }
    bool flag() { // compute_grad_*
        if (!ok || at >= n || !PyBool_Check(args[at])) {
            ok = false;
            return false;
        }
        return args[at++] == Py_True;
    }
    const Tensor* fail() {
        ok = false;
        return nullptr;
    }
};

// Runs `body` (which returns the status of a C ABI call) for the device of `like` on torch's
// current stream.
template <typename F> int on_stream_of(const Tensor& like, F&& body) {
    const c10::cuda::CUDAGuard guard(like.device());
    void* previous = mops_b200_get_stream();
    mops_b200_set_stream(at::cuda::getCurrentCUDAStream().stream());
    int status;
    Py_BEGIN_ALLOW_THREADS;
    status = body();
    Py_END_ALLOW_THREADS;
    mops_b200_set_stream(previous);
    return status;
}

PyObject* raise(int status) {
    PyObject* error = PyObject_CallFunction(g_error, "si", mops_get_last_error_message(), status);
    if (error != nullptr) {
        PyErr_SetObject(g_error, error);
        Py_DECREF(error);
    }
    return nullptr;
}

PyObject* wrap(const Tensor& t) {
    if (!t.defined()) Py_RETURN_NONE;
    return THPVariable_Wrap(t);
}
PyObject* wrap(std::initializer_list<Tensor> ts) {
    PyObject* tuple = PyTuple_New(static_cast<Py_ssize_t>(ts.size()));
    Py_ssize_t i = 0;
    for (const Tensor& t : ts) PyTuple_SET_ITEM(tuple, i++, wrap(t));
    return tuple;
}

Tensor like(const Tensor* t, bool want) { return want ? at::empty(t->sizes(), t->options()) : Tensor(); }

#define CALL(NAME, ...)                                                                            \
    on_stream_of(*args.first, [&] {                                                                \
        return args.first->scalar_type() == at::kDouble ? mops_cuda_##NAME##_f64(__VA_ARGS__)      \
                                                        : mops_cuda_##NAME##_f32(__VA_ARGS__);     \
    })
#define READY                                                                                      \
    if (!args.ok || args.at != args.n) Py_RETURN_NOTIMPLEMENTED

PyObject* hpe(Args& args) {
    auto A = args.real(2), C = args.real(1), P = args.index(2);
    READY;
    Tensor out = at::empty({A->size(0)}, A->options());
    const int status = CALL(homogeneous_polynomial_evaluation, Arg{&out}, Arg{A}, Arg{C}, Arg{P});
    return status != 0 ? raise(status) : wrap(out);
}
PyObject* hpe_vjp(Args& args) {
    auto g = args.real(1), A = args.real(2), C = args.real(1), P = args.index(2);
    const bool want = args.flag();
    READY;
    Tensor gA = like(A, want);
    const int status = CALL(homogeneous_polynomial_evaluation_vjp, Arg{&gA}, Arg{g}, Arg{A}, Arg{C}, Arg{P});
    return status != 0 ? raise(status) : wrap(gA);
}
PyObject* sap(Args& args) {
    auto A = args.real(2), B = args.real(2), C = args.real(1), PA = args.index(1), PB = args.index(1),
         PO = args.index(1);
    const int64_t nO = args.size();
    READY;
    Tensor out = at::empty({A->size(0), nO}, A->options());
    const int status = CALL(sparse_accumulation_of_products, Arg{&out}, Arg{A}, Arg{B}, Arg{C}, Arg{PA},
                            Arg{PB}, Arg{PO});
    return status != 0 ? raise(status) : wrap(out);
}
PyObject* sap_vjp(Args& args) {
    auto g = args.real(2), A = args.real(2), B = args.real(2), C = args.real(1), PA = args.index(1),
         PB = args.index(1), PO = args.index(1);
    const bool want_A = args.flag(), want_B = args.flag();
    READY;
    Tensor gA = like(A, want_A), gB = like(B, want_B);
    const int status = CALL(sparse_accumulation_of_products_vjp, Arg{&gA}, Arg{&gB}, Arg{g}, Arg{A}, Arg{B},
                            Arg{C}, Arg{PA}, Arg{PB}, Arg{PO});
    return status != 0 ? raise(status) : wrap({gA, gB});
}
PyObject* opsa(Args& args) {
    auto A = args.real(2), B = args.real(2), P = args.index(1);
    const int64_t nO = args.size();
    READY;
    Tensor out = at::empty({nO, A->size(1), B->size(1)}, A->options());
    const int status = CALL(outer_product_scatter_add, Arg{&out}, Arg{A}, Arg{B}, Arg{P});
    return status != 0 ? raise(status) : wrap(out);
}
PyObject* opsa_vjp(Args& args) {
    auto g = args.real(3), A = args.real(2), B = args.real(2), P = args.index(1);
    const bool want_A = args.flag(), want_B = args.flag();
    READY;
    Tensor gA = like(A, want_A), gB = like(B, want_B);
    const int status = CALL(outer_product_scatter_add_vjp, Arg{&gA}, Arg{&gB}, Arg{g}, Arg{A}, Arg{B}, Arg{P});
    return status != 0 ? raise(status) : wrap({gA, gB});
}
PyObject* opsaw(Args& args) {
    auto A = args.real(2), B = args.real(2), W = args.real(2), PW = args.index(1), PO = args.index(1);
    READY;
    Tensor out = at::empty({W->size(0), A->size(1), B->size(1)}, A->options());
    const int status =
        CALL(outer_product_scatter_add_with_weights, Arg{&out}, Arg{A}, Arg{B}, Arg{W}, Arg{PW}, Arg{PO});
    return status != 0 ? raise(status) : wrap(out);
}
PyObject* opsaw_vjp(Args& args) {
    auto g = args.real(3), A = args.real(2), B = args.real(2), W = args.real(2), PW = args.index(1),
         PO = args.index(1);
    const bool want_A = args.flag(), want_B = args.flag(), want_W = args.flag();
    READY;
    Tensor gA = like(A, want_A), gB = like(B, want_B), gW = like(W, want_W);
    const int status = CALL(outer_product_scatter_add_with_weights_vjp, Arg{&gA}, Arg{&gB}, Arg{&gW}, Arg{g},
                            Arg{A}, Arg{B}, Arg{W}, Arg{PW}, Arg{PO});
    return status != 0 ? raise(status) : wrap({gA, gB, gW});
}
PyObject* sasaw(Args& args) {
    auto A = args.real(2), B = args.real(2), C = args.real(1), W = args.real(3), M1 = args.index(1),
         J = args.index(1), M2 = args.index(1), I = args.index(1), M3 = args.index(1);
    const int64_t nO = args.size();
    READY;
    Tensor out = at::empty({W->size(0), nO, B->size(1)}, A->options());
    const int status = CALL(sparse_accumulation_scatter_add_with_weights, Arg{&out}, Arg{A}, Arg{B}, Arg{C},
                            Arg{W}, Arg{M1}, Arg{J}, Arg{M2}, Arg{I}, Arg{M3});
    return status != 0 ? raise(status) : wrap(out);
}
PyObject* sasaw_vjp(Args& args) {
    auto g = args.real(3), A = args.real(2), B = args.real(2), C = args.real(1), W = args.real(3),
         M1 = args.index(1), J = args.index(1), M2 = args.index(1), I = args.index(1), M3 = args.index(1);
    const bool want_A = args.flag(), want_B = args.flag(), want_W = args.flag();
    READY;
    Tensor gA = like(A, want_A), gB = like(B, want_B), gW = like(W, want_W);
    const int status =
        CALL(sparse_accumulation_scatter_add_with_weights_vjp, Arg{&gA}, Arg{&gB}, Arg{&gW}, Arg{g}, Arg{A},
             Arg{B}, Arg{C}, Arg{W}, Arg{M1}, Arg{J}, Arg{M2}, Arg{I}, Arg{M3});
    return status != 0 ? raise(status) : wrap({gA, gB, gW});
}

PyObject* (*const kOperations[])(Args&) = {hpe,      hpe_vjp, sap,       sap_vjp, opsa,
                                           opsa_vjp, opsaw,   opsaw_vjp, sasaw,   sasaw_vjp};

PyObject* call(PyObject*, PyObject* const* args, Py_ssize_t n) {
    const long which = n > 0 ? PyLong_AsLong(args[0]) : -1;
    if (which < 0 || which >= static_cast<long>(sizeof(kOperations) / sizeof(kOperations[0]))) {
        PyErr_Clear();
        Py_RETURN_NOTIMPLEMENTED;
    }
    Args rest{args + 1, n - 1};
    HANDLE_TH_ERRORS // (allocation of the results: torch.OutOfMemoryError, as from Python)
    return kOperations[which](rest);
    END_HANDLE_TH_ERRORS
}

PyObject* setup(PyObject*, PyObject* error) {
    Py_XSETREF(g_error, Py_NewRef(error));
    Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"call", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(call)), METH_FASTCALL,
     "call(operation, arguments...): results, or NotImplemented"},
    {"setup", setup, METH_O, "setup(error): the exception to raise"},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_calls", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

} // namespace

PyMODINIT_FUNC PyInit__calls() { return PyModule_Create(&kModule); }
