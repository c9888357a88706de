// Python entry points of the kernel-level operators (ops.py): tensors to the C ABI in one native step.
//
// A small operator call is bound by its host work.  Through Python and ctypes (a Stream object, an output by
// keyword arguments, twenty converted arguments) dcvc_conv1x1 of 390 x 768 x 768 takes 13.9 us for 5 us of
// GPU time, of which the library itself, tensor maps and launch, needs 4.  These functions read the tensors'
// fields, allocate the output and ask for the stream in C++ and call the library directly: 4.5 us
// (dcvc_conv_ffn of 1000 x 256 13.4 -> 6.3, dcvc_dwconv3x3 of 8 x 8 x 256 10.4 -> 4.1).
//
// Each takes positional arguments (None for an absent tensor) and returns the output tensor, or the
// library's status as an int when it is not 0.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "dcvc_b200.h"

namespace {

// The argument errors of the Python wrappers these stand in for.
struct CallError {
    PyObject* type;
    const char* text;
};

const at::Tensor& tensor(PyObject* o)
{
    if (!THPVariable_Check(o)) {
        throw CallError{PyExc_TypeError, "a torch.Tensor is required"};
    }
    return THPVariable_Unpack(o);
}

int integer(PyObject* o)
{
    const long v = PyLong_AsLong(o);
    if (v == -1 && PyErr_Occurred() != nullptr) {
        throw CallError{nullptr, nullptr};
    }
    return static_cast<int>(v);
}

// One optional tensor: its data and row pitch, null and 0 when absent.
struct Opt {
    void* p = nullptr;
    int ld = 0;
};

void* data(PyObject* o) { return o == Py_None ? nullptr : tensor(o).data_ptr(); }

Opt rows(PyObject* o)
{
    if (o == Py_None) {
        return {};
    }
    const at::Tensor& t = tensor(o);
    return {t.data_ptr(), static_cast<int>(t.stride(0))};
}

void require(bool ok, const char* text)
{
    if (!ok) {
        throw CallError{PyExc_AssertionError, text};
    }
}

int dtype_code(const at::Tensor& t)
{
    switch (t.scalar_type()) {
    case at::kHalf: return DCVC_F16;
    case at::kBFloat16: return DCVC_BF16;
    default: throw CallError{PyExc_KeyError, "the dtype must be torch.float16 or torch.bfloat16"};
    }
}

at::Tensor output(PyObject* out, const at::Tensor& like, at::IntArrayRef shape, at::ScalarType type)
{
    return out != Py_None ? tensor(out) : at::empty(shape, like.options().dtype(type));
}

void* current_stream() { return c10::cuda::getCurrentCUDAStream(c10::cuda::current_device()).stream(); }

// The library call without the GIL, then the output or the status.
template <typename F>
PyObject* finish(const at::Tensor& out, F&& call)
{
    int status = 0;
    Py_BEGIN_ALLOW_THREADS
    status = call();
    Py_END_ALLOW_THREADS
    return status == 0 ? THPVariable_Wrap(out) : PyLong_FromLong(status);
}

template <Py_ssize_t COUNT, typename F>
PyObject* guarded(Py_ssize_t n, F&& body)
{
    if (n != COUNT) {
        PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", COUNT, n);
        return nullptr;
    }
    HANDLE_TH_ERRORS
    try {
        return body();
    } catch (const CallError& e) {
        if (e.type != nullptr) {
            PyErr_SetString(e.type, e.text);
        }
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
}

// (a, w, bias, epilogue, res, res2, qscale, out, sub_w, sub_cout, block_n)
PyObject* conv1x1(PyObject*, PyObject* const* v, Py_ssize_t n)
{
    return guarded<11>(n, [&]() -> PyObject* {
        const at::Tensor &a = tensor(v[0]), &w = tensor(v[1]);
        require(a.dim() == 2 && a.stride(1) == 1 && w.is_contiguous(), "a [M, K] with unit columns, w contiguous");
        const int epi = integer(v[3]), sub_w = integer(v[8]), sub_cout = integer(v[9]), block_n = integer(v[10]);
        const int64_t M = a.size(0), K = a.size(1), N = w.size(0);
        const int64_t om = epi == DCVC_EPI_SUBPEL ? 4 * M : M;
        const int64_t on = epi == DCVC_EPI_QUAD ? N / 4 : epi == DCVC_EPI_SUBPEL ? sub_cout : N;
        const int dtype = dtype_code(a);
        const at::Tensor out = output(v[7], a, {om, on}, a.scalar_type());
        const Opt res = rows(v[4]), res2 = rows(v[5]);
        const float* bias = static_cast<const float*>(data(v[2]));
        const void *q = data(v[6]), *ap = a.data_ptr(), *wp = w.data_ptr();
        void* op = out.data_ptr();
        const int lda = static_cast<int>(a.stride(0)), ldo = static_cast<int>(out.stride(0));
        void* s = current_stream();
        return finish(out, [&] {
            return dcvc_conv1x1(dtype, epi, static_cast<int>(M), static_cast<int>(N), static_cast<int>(K), ap, lda, wp, bias, res.p,
                                res.ld, res2.p, res2.ld, q, op, ldo, sub_w, sub_cout, block_n, s);
        });
    });
}

// (a, w, wscale, bias, epilogue, out, block_n)
PyObject* conv1x1_f8(PyObject*, PyObject* const* v, Py_ssize_t n)
{
    return guarded<7>(n, [&]() -> PyObject* {
        const at::Tensor &a = tensor(v[0]), &w = tensor(v[1]);
        require(a.dim() == 2 && a.stride(1) == 1 && w.is_contiguous(), "a [M, K] with unit columns, w contiguous");
        const int epi = integer(v[4]), block_n = integer(v[6]);
        const int64_t M = a.size(0), K = a.size(1), N = w.size(0);
        const at::Tensor out = output(v[5], a, {M, epi == DCVC_EPI_QUAD ? N / 4 : N}, at::kBFloat16);
        const void *ap = a.data_ptr(), *wp = w.data_ptr();
        const float *ws = static_cast<const float*>(tensor(v[2]).data_ptr()), *bias = static_cast<const float*>(tensor(v[3]).data_ptr());
        void* op = out.data_ptr();
        const int lda = static_cast<int>(a.stride(0)), ldo = static_cast<int>(out.stride(0));
        void* s = current_stream();
        return finish(out, [&] {
            return dcvc_conv1x1_f8(epi, static_cast<int>(M), static_cast<int>(N), static_cast<int>(K), ap, lda, wp, ws, bias, op, ldo,
                                   block_n, s);
        });
    });
}

// (x, w1, b1, w2, b2, qscale, out, block_n)
PyObject* conv_ffn(PyObject*, PyObject* const* v, Py_ssize_t n)
{
    return guarded<8>(n, [&]() -> PyObject* {
        const at::Tensor &x = tensor(v[0]), &w1 = tensor(v[1]), &w2 = tensor(v[3]);
        require(x.dim() == 2 && x.stride(1) == 1 && w1.is_contiguous() && w2.is_contiguous(),
                "x [M, C] with unit columns, w1 and w2 contiguous");
        const int block_n = integer(v[7]);
        const int64_t M = x.size(0), C = x.size(1), F = w2.size(1);
        const at::Tensor out = output(v[6], x, {M, C}, x.scalar_type());
        const void *xp = x.data_ptr(), *w1p = w1.data_ptr(), *w2p = w2.data_ptr(), *q = data(v[5]);
        const float *b1 = static_cast<const float*>(tensor(v[2]).data_ptr()), *b2 = static_cast<const float*>(tensor(v[4]).data_ptr());
        void* op = out.data_ptr();
        const int ldx = static_cast<int>(x.stride(0)), ldo = static_cast<int>(out.stride(0));
        void* s = current_stream();
        const long long ws = block_n == 0 ? dcvc_conv_ffn_workspace(static_cast<int>(M), static_cast<int>(C), static_cast<int>(F)) : 0;
        if (ws > 0) {
            // from the caching allocator, as the output: reused only behind this call's work on the stream
            const at::Tensor t = at::empty({M, F}, x.options());
            void* tp = t.data_ptr();
            const long long bytes = static_cast<long long>(t.nbytes());
            return finish(out, [&] {
                return dcvc_conv_ffn_ws(static_cast<int>(M), static_cast<int>(C), static_cast<int>(F), xp, ldx, w1p, b1, w2p, b2, q,
                                        op, ldo, tp, bytes, s);
            });
        }
        return finish(out, [&] {
            return dcvc_conv_ffn(static_cast<int>(M), static_cast<int>(C), static_cast<int>(F), xp, ldx, w1p, b1, w2p, b2, q, op, ldo,
                                 block_n, s);
        });
    });
}

// (x, H, W, w, img_h, out); `ex`: FP16 or BF16 and stacked images, else dcvc_dwconv3x3
PyObject* dwconv(PyObject* const* v, Py_ssize_t n, bool ex)
{
    return guarded<6>(n, [&]() -> PyObject* {
        const at::Tensor &x = tensor(v[0]), &w = tensor(v[3]);
        const int H = integer(v[1]), W = integer(v[2]), img_h = integer(v[4]);
        const int C = static_cast<int>(x.size(1));
        const at::Tensor out = v[5] != Py_None ? tensor(v[5]) : at::empty_like(x);
        const int dtype = ex ? dtype_code(x) : DCVC_F16;
        const void* xp = x.data_ptr();
        const float* wp = static_cast<const float*>(w.data_ptr());
        void* op = out.data_ptr();
        const int ldx = static_cast<int>(x.stride(0)), ldo = static_cast<int>(out.stride(0));
        void* s = current_stream();
        return finish(out, [&] {
            return ex ? dcvc_dwconv3x3_ex(dtype, xp, H, W, img_h, C, ldx, wp, op, ldo, s)
                      : dcvc_dwconv3x3(xp, H, W, C, ldx, wp, op, ldo, s);
        });
    });
}

PyObject* dwconv3x3(PyObject*, PyObject* const* v, Py_ssize_t n) { return dwconv(v, n, false); }
PyObject* dwconv3x3_ex(PyObject*, PyObject* const* v, Py_ssize_t n) { return dwconv(v, n, true); }

template <typename F>
PyMethodDef method(const char* name, F f)
{
    return {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL, nullptr};
}

PyMethodDef methods[] = {method("conv1x1", conv1x1),     method("conv1x1_f8", conv1x1_f8),     method("conv_ffn", conv_ffn),
                         method("dwconv3x3", dwconv3x3), method("dwconv3x3_ex", dwconv3x3_ex), {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_torch_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__torch_calls() { return PyModule_Create(&module); }
