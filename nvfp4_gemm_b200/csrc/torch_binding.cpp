// CPython module between torch tensors and the C ABI (include/nvfp4_b200.h): turns the operator's
// 7-tuple (template.py:9-18 in the reference project) into struct nvfp4_problem and makes the call on
// torch's current stream.
//
// What bounds a small matmul is the time to issue it: the kernel launch itself takes the CPU
// 2.3-2.5 us.  The translation reads about forty sizes and strides; through Python attributes and
// ctypes a call took 11-12 us (128 x 256 x 256: 10.3 us a pass although the kernel runs for 3.3 us),
// and a table of translated tuples by address does not help a caller whose tensors are new.  From C++
// the same reads take well under a microsecond, so nothing is remembered between calls (128 x 256 x 256:
// 3.75 us a pass; a first call on new tensors 28.5 -> 17.6 us, waited for).
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>
#include <exception>

#include "../../include/nvfp4_b200.h"

namespace {

struct PythonError {};   // a Python exception is set

[[noreturn]] void raise(PyObject* type, const char* text) {
    PyErr_SetString(type, text);
    throw PythonError{};
}

// A tensor of the tuple, or null for None.
const at::Tensor* tensor_or_none(PyObject* o) {
    if (o == Py_None) return nullptr;
    if (!THPVariable_Check(o)) {
        PyErr_Format(PyExc_TypeError, "expected a tensor, got %s", Py_TYPE(o)->tp_name);
        throw PythonError{};
    }
    return &THPVariable_Unpack(o);
}

int64_t batch_stride(const at::Tensor& t, int64_t dim) {
    if (t.dim() <= dim) raise(PyExc_IndexError, "tensor has no batch dimension");
    return t.size(dim) > 1 ? t.stride(dim) : 0;
}

struct Operands {
    PyObject* seq;            // keeps the tensors alive
    const at::Tensor* t[7];   // a, b, sfa, sfb, sfa_permuted, sfb_permuted, c; the last five may be null
    explicit Operands(PyObject* data) : seq(PySequence_Fast(data, "expected (a, b, sfa, sfb, sfa_permuted, sfb_permuted, c)")) {
        if (!seq) throw PythonError{};
        try {
            if (PySequence_Fast_GET_SIZE(seq) != 7) raise(PyExc_ValueError, "expected seven values: (a, b, sfa, sfb, sfa_permuted, sfb_permuted, c)");
            for (int i = 0; i < 7; ++i) t[i] = tensor_or_none(PySequence_Fast_GET_ITEM(seq, i));
            if (!t[0] || !t[1]) raise(PyExc_TypeError, "a and b must be tensors");
        } catch (const PythonError&) {
            Py_DECREF(seq);
            throw;
        }
    }
    ~Operands() { Py_DECREF(seq); }
    Operands(const Operands&) = delete;
    Operands& operator=(const Operands&) = delete;
    void require_cuda() const {
        for (const at::Tensor* x : t)
            if (x && !x->is_cuda()) raise(PyExc_ValueError, "custom_kernel needs CUDA tensors (there is no CPU fallback)");
    }
};

nvfp4_problem make_problem(const Operands& o) {
    const at::Tensor &a = *o.t[0], &b = *o.t[1];
    const at::Tensor* c = o.t[6];
    if (a.dim() != 3 || b.dim() != 3 || (c && c->dim() != 3)) raise(PyExc_ValueError, "a, b and c must have three dimensions (rows, columns, batch)");
    const int64_t m = a.size(0), k_bytes = a.size(1), l = a.size(2), n = b.size(0);
    if (b.size(1) != k_bytes || b.size(2) != l) {
        PyErr_Format(PyExc_ValueError, "a (%lld, %lld, %lld) and b (%lld, %lld, %lld) disagree on k or l", (long long)m, (long long)k_bytes,
                     (long long)l, (long long)n, (long long)b.size(1), (long long)b.size(2));
        throw PythonError{};
    }
    if (c && (c->size(0) != m || c->size(1) != n || c->size(2) != l)) {
        PyErr_Format(PyExc_ValueError, "c has shape (%lld, %lld, %lld), expected (%lld, %lld, %lld)", (long long)c->size(0), (long long)c->size(1),
                     (long long)c->size(2), (long long)m, (long long)n, (long long)l);
        throw PythonError{};
    }
    if (m > INT32_MAX || n > INT32_MAX || k_bytes > INT32_MAX / 2 || l > INT32_MAX) raise(PyExc_ValueError, "sizes must fit 32 bits");
    if (a.stride(1) != 1 || b.stride(1) != 1 || (c && c->stride(1) != 1 && n > 1))
        raise(PyExc_ValueError, "a, b must be K-major (stride 1 along k) and c row-major");
    bool types = a.element_size() == 1 && b.element_size() == 1 && (!c || c->scalar_type() == at::kHalf);
    for (int i = 2; i < 6; ++i) types = types && (!o.t[i] || o.t[i]->element_size() == 1);
    if (!types) raise(PyExc_ValueError, "expected packed fp4 (1 byte per 2 values), 1-byte scales and fp16 output");

    nvfp4_problem p;
    std::memset(&p, 0, sizeof(p));
    p.a = a.data_ptr();
    p.b = b.data_ptr();
    p.c = c ? c->data_ptr() : nullptr;
    p.m = static_cast<int32_t>(m);
    p.n = static_cast<int32_t>(n);
    p.k = static_cast<int32_t>(2 * k_bytes);
    p.l = static_cast<int32_t>(l);
    p.a_row_stride = a.stride(0);
    p.a_batch_stride = batch_stride(a, 2);
    p.b_row_stride = n > 1 ? b.stride(0) : k_bytes;
    p.b_batch_stride = batch_stride(b, 2);
    if (const at::Tensor* s = o.t[2]) {
        p.sfa = s->data_ptr();
        p.sfa_batch_stride = batch_stride(*s, 2);
        p.sfa_row_stride = s->stride(0);
    }
    if (const at::Tensor* s = o.t[3]) {
        p.sfb = s->data_ptr();
        p.sfb_batch_stride = batch_stride(*s, 2);
        p.sfb_row_stride = n > 1 ? s->stride(0) : k_bytes / 8;
    }
    // permuted scales: [32, 4, rest_rows, 4, rest_k, L]; the batch is the last dimension
    if (const at::Tensor* s = o.t[4]) {
        p.sfa_perm = s->data_ptr();
        p.sfa_perm_batch_stride = batch_stride(*s, 5);
    }
    if (const at::Tensor* s = o.t[5]) {
        p.sfb_perm = s->data_ptr();
        p.sfb_perm_batch_stride = batch_stride(*s, 5);
    }
    if (c) {
        p.c_row_stride = c->stride(0);
        p.c_batch_stride = batch_stride(*c, 2);
    }
    return p;
}

// Calls f(stream) with the tensors' device current, on torch's current stream of that device and
// without the interpreter lock (a launch waits when the queue of the device is full).  Only f, which
// answers with a status, runs unlocked: the guard and the stream throw where CUDA reports an error, and
// an exception that left with the lock released would be turned into a Python one without a thread state.
template <class F>
int on_current_stream(const at::Tensor& a, F f) {
    const c10::DeviceIndex dev = a.device().index();
    const c10::cuda::CUDAGuard guard(dev);
    void* stream = c10::cuda::getCurrentCUDAStream(dev).stream();
    int rc = 0;
    Py_BEGIN_ALLOW_THREADS
    rc = f(stream);
    Py_END_ALLOW_THREADS
    return rc;
}

template <class F>
PyObject* guarded(F f) {
    try {
        return f();
    } catch (const PythonError&) {
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
    }
    return nullptr;
}

// matmul(data) -> status of nvfp4_matmul
PyObject* py_matmul(PyObject*, PyObject* data) {
    return guarded([&] {
        const Operands o(data);
        o.require_cuda();
        const nvfp4_problem p = make_problem(o);
        return PyLong_FromLong(on_current_stream(*o.t[0], [&](void* stream) { return nvfp4_matmul(&p, stream); }));
    });
}

// fill_problem(data, address): writes struct nvfp4_problem at `address`
PyObject* py_fill_problem(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 2) raise(PyExc_TypeError, "fill_problem(data, address)");
        void* dst = PyLong_AsVoidPtr(args[1]);
        if (!dst) {
            if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "address is NULL");
            throw PythonError{};
        }
        const nvfp4_problem p = make_problem(Operands(args[0]));
        std::memcpy(dst, &p, sizeof(p));
        Py_RETURN_NONE;
    });
}

int int_arg(PyObject* o) {
    const long v = PyLong_AsLong(o);
    if (v == -1 && PyErr_Occurred()) throw PythonError{};
    if (v < INT32_MIN || v > INT32_MAX) raise(PyExc_OverflowError, "argument does not fit 32 bits");
    return static_cast<int>(v);
}

// gemm_epilogue(data, bias, activation, out, tile_n, grid, cta_group, split_k) -> status of
// nvfp4_gemm_epilogue.  out: None for fp16 into data[6], else (packed, sf, sf_permuted) with dense rows.
PyObject* py_gemm_epilogue(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    return guarded([&] {
        if (nargs != 8) raise(PyExc_TypeError, "gemm_epilogue(data, bias, activation, out, tile_n, grid, cta_group, split_k)");
        const Operands o(args[0]);
        o.require_cuda();
        if (args[3] == Py_None && !o.t[6]) raise(PyExc_ValueError, "an fp16 output needs data[6]");
        const nvfp4_problem p = make_problem(o);
        nvfp4_epilogue e;
        std::memset(&e, 0, sizeof(e));
        if (const at::Tensor* bias = tensor_or_none(args[1])) {
            if (bias->scalar_type() != at::kHalf || bias->numel() != p.n || !bias->is_contiguous())
                raise(PyExc_ValueError, "bias must be a contiguous fp16 vector of length n");
            e.bias = bias->data_ptr();
        }
        e.activation = int_arg(args[2]);
        if (args[3] != Py_None) {
            struct Sequence {          // any sequence will do
                PyObject* seq;
                ~Sequence() { Py_XDECREF(seq); }
            } const out{PySequence_Fast(args[3], "out must be (packed, sf, sf_permuted)")};
            if (!out.seq) throw PythonError{};
            if (PySequence_Fast_GET_SIZE(out.seq) < 3) raise(PyExc_IndexError, "out must be (packed, sf, sf_permuted)");
            void* ptr[3];
            for (int i = 0; i < 3; ++i) {
                const at::Tensor* t = tensor_or_none(PySequence_Fast_GET_ITEM(out.seq, i));
                if (!t) raise(PyExc_TypeError, "out must be (packed, sf, sf_permuted)");
                ptr[i] = t->data_ptr();
            }
            const int64_t m = p.m, n = p.n;
            e.output = NVFP4_OUT_NVFP4;
            e.out_packed = ptr[0];
            e.out_sf = ptr[1];
            e.out_sf_perm = ptr[2];
            e.out_packed_row_stride = n / 2;
            e.out_packed_batch_stride = m * (n / 2);
            e.out_sf_row_stride = n / 16;
            e.out_sf_batch_stride = m * (n / 16);
            e.out_sf_perm_batch_stride = ((m + 127) / 128) * (n / 64) * 512;
        }
        nvfp4_gemm_config cfg = {int_arg(args[4]), 0, int_arg(args[5]), int_arg(args[6]), int_arg(args[7]), 0};
        return PyLong_FromLong(on_current_stream(*o.t[0], [&](void* stream) { return nvfp4_gemm_epilogue(&p, &cfg, &e, stream); }));
    });
}

// Read from the file by nvfp4_gemm_b200/build.py: the types of torch and Python that this code has the layouts of.
[[gnu::used]] const char built_for[] = "nvfp4_native built for: " NVFP4_BUILT_FOR;

PyMethodDef methods[] = {
    {"matmul", py_matmul, METH_O, "matmul(data) -> status"},
    {"fill_problem", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_fill_problem)), METH_FASTCALL, "fill_problem(data, address)"},
    {"gemm_epilogue", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_gemm_epilogue)), METH_FASTCALL,
     "gemm_epilogue(data, bias, activation, out, tile_n, grid, cta_group, split_k) -> status"},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", "torch tensors to the C ABI of libnvfp4_b200", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() { return PyModule_Create(&module); }
