// Python calls of single operators on torch tensors (functional.py) without ctypes.
//
// A layer of a small network is a handful of launches of a few microseconds each, and what its caller waits for is the host:
// through ctypes one call cost 7 us - attribute reads and checks of every tensor, the descriptor, torch.empty, argument
// conversion - where the launch itself takes 2.  Here a call is: unpack, check, describe, allocate the result, launch.
// Forward, three gradients and the fused epilogue of a 12 x 20 x 36 -> 40 layer: 17 us, 37 through ctypes.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstring>
#include <unordered_map>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "dcgan_b200.h"

namespace {

struct Error {};   // a Python exception is set

[[noreturn]] void fail(PyObject* type, const char* message)
{
    PyErr_SetString(type, message);
    throw Error();
}

PyObject* g_check = nullptr;      // _lib.check: raises DcgError for a status
PyObject* g_epilogue = nullptr;   // _lib.Epilogue

const at::Tensor& tensor(PyObject* o)
{
    if (!THPVariable_Check(o)) fail(PyExc_AssertionError, "expected a torch tensor");
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.is_cuda() || !t.is_contiguous() || t.scalar_type() != at::kFloat)
        fail(PyExc_AssertionError, "expected a contiguous float32 CUDA tensor");
    return t;
}
const at::Tensor& tensor4(PyObject* o)
{
    const at::Tensor& t = tensor(o);
    if (t.dim() != 4) fail(PyExc_ValueError, "expected four dimensions");
    return t;
}
float* pointer(PyObject* o) { return o == Py_None ? nullptr : static_cast<float*>(tensor(o).data_ptr()); }

int to_int(PyObject* o)
{
    const long v = PyLong_AsLong(o);
    if (v == -1 && PyErr_Occurred()) throw Error();
    return (int)v;
}
float to_float(PyObject* o)
{
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw Error();
    return (float)v;
}

void pair(PyObject* o, int& a, int& b)
{
    if (PyTuple_CheckExact(o) && PyTuple_GET_SIZE(o) == 2) {
        a = to_int(PyTuple_GET_ITEM(o, 0));
        b = to_int(PyTuple_GET_ITEM(o, 1));
        return;
    }
    PyObject* seq = PySequence_Tuple(o);
    if (!seq) throw Error();
    const bool two = PyTuple_GET_SIZE(seq) >= 2;
    if (two) {
        a = (int)PyLong_AsLong(PyTuple_GET_ITEM(seq, 0));
        b = (int)PyLong_AsLong(PyTuple_GET_ITEM(seq, 1));
    }
    Py_DECREF(seq);
    if (PyErr_Occurred()) throw Error();
    if (!two) fail(PyExc_ValueError, "expected a pair");
}

// The geometry functional.conv_desc describes: `pad` is the total pad, SAME where None (src/ops/conv2d.cu:33-41); the output
// is (in + pad - k) / stride + 1 where not given.
int same_pad(int in, int k, int s)
{
    const int p = in % s == 0 ? k - s : k - in % s;
    return p > 0 ? p : 0;
}
int floor_div(int a, int b) { return a / b - (a % b != 0 && (a < 0) != (b < 0)); }

dcg_conv_desc describe(int n, int h, int w, int c, int kh, int kw, int o, PyObject* strides, PyObject* pad, PyObject* out_hw)
{
    dcg_conv_desc d{};
    d.n = n; d.h = h; d.w = w; d.c = c; d.kh = kh; d.kw = kw; d.o = o;
    pair(strides, d.stride_h, d.stride_w);
    if (d.stride_h == 0 || d.stride_w == 0) fail(PyExc_ZeroDivisionError, "stride of zero");
    int ph, pw;
    if (pad == Py_None) {
        ph = same_pad(h, kh, d.stride_h);
        pw = same_pad(w, kw, d.stride_w);
    } else {
        pair(pad, ph, pw);
    }
    if (out_hw == Py_None) {
        d.ho = floor_div(h + ph - kh, d.stride_h) + 1;
        d.wo = floor_div(w + pw - kw, d.stride_w) + 1;
    } else {
        pair(out_hw, d.ho, d.wo);
    }
    d.pad_top = floor_div(ph, 2);
    d.pad_left = floor_div(pw, 2);
    return d;
}

// Scratch bytes of a call.  Working them out plans the convolution, so they are kept per descriptor (a bounded table).
struct CallKey {
    int v[15];
    bool operator==(const CallKey& o) const { return memcmp(v, o.v, sizeof v) == 0; }
};
struct CallHash {
    size_t operator()(const CallKey& k) const
    {
        size_t h = 1469598103934665603ull;
        for (int i : k.v) h = (h ^ (unsigned)i) * 1099511628211ull;
        return h;
    }
};
size_t conv_scratch(const dcg_conv_desc& d, int kind, int precision)
{
    static std::unordered_map<CallKey, size_t, CallHash> table;   // under the GIL
    CallKey key;
    static_assert(sizeof(dcg_conv_desc) == 13 * sizeof(int), "the descriptor is 13 ints");
    memcpy(key.v, &d, sizeof d);
    key.v[13] = kind; key.v[14] = precision;
    const auto it = table.find(key);
    if (it != table.end()) return it->second;
    if (table.size() >= 1024) table.clear();
    return table[key] = dcg_conv_workspace_bytes(&d, kind, precision);
}

at::Tensor new_tensor(at::IntArrayRef shape, at::ScalarType type, c10::Device device)
{
    return at::detail::empty_cuda(shape, type, device, std::nullopt);
}
// The scratch of one call, from torch's caching allocator: held until the launches have been enqueued, and then only the same
// stream gets the memory again.  A buffer kept for the next call would be shared by all streams and threads (kernels of two
// streams would write the same partial tiles), and growing it would take it from under kernels and captured graphs that use it.
struct Scratch {
    at::Tensor memory;
    size_t bytes;
    Scratch(size_t need, c10::Device device) : bytes(need)
    {
        if (need) memory = new_tensor({(int64_t)need}, at::kByte, device);
    }
    void* data() const { return bytes ? memory.data_ptr() : nullptr; }
};

void check(int status)
{
    if (status == DCG_OK) return;
    PyObject* r = PyObject_CallFunction(g_check, "i", status);
    Py_XDECREF(r);
    if (!r) throw Error();
    fail(PyExc_RuntimeError, "operator failed");
}

// A ctypes Epilogue exposes its memory through the buffer protocol.
struct EpilogueView {
    Py_buffer view{};
    const dcg_epilogue* ep = nullptr;
    explicit EpilogueView(PyObject* o, int flags = PyBUF_SIMPLE)
    {
        if (o == Py_None) return;
        const int is_one = PyObject_IsInstance(o, g_epilogue);
        if (is_one < 0) throw Error();
        if (!is_one) fail(PyExc_TypeError, "expected an Epilogue");
        if (PyObject_GetBuffer(o, &view, flags) != 0) throw Error();
        if ((size_t)view.len != sizeof(dcg_epilogue)) { PyBuffer_Release(&view); fail(PyExc_TypeError, "expected an Epilogue"); }
        ep = static_cast<const dcg_epilogue*>(view.buf);
    }
    ~EpilogueView() { if (ep) PyBuffer_Release(&view); }
};

// kind: which of the operators; a, b: its operands; desc complete.  Returns the result as a new reference.
PyObject* run_conv(int kind, const dcg_conv_desc& d, const at::Tensor& a, const at::Tensor& b, PyObject* epilogue, int precision, PyObject* out)
{
    const size_t need = conv_scratch(d, kind, precision);
    const c10::Device device = a.device();
    at::Tensor result;
    float* dst;
    if (out == Py_None) {
        const int64_t shapes[3][4] = {{d.n, d.ho, d.wo, d.o}, {d.n, d.h, d.w, d.c}, {d.kh, d.kw, d.c, d.o}};
        result = new_tensor(at::IntArrayRef(shapes[kind], 4), at::kFloat, device);
        dst = static_cast<float*>(result.data_ptr());
    } else {
        dst = static_cast<float*>(tensor(out).data_ptr());
    }
    const Scratch ws(need, device);
    const EpilogueView ep(epilogue);
    const float *pa = static_cast<const float*>(a.data_ptr()), *pb = static_cast<const float*>(b.data_ptr());
    void* stream = c10::cuda::getCurrentCUDAStream().stream();
    int status;
    Py_BEGIN_ALLOW_THREADS
    if (kind == 0) status = dcg_conv2d_fwd(&d, pa, pb, dst, ep.ep, precision, ws.data(), ws.bytes, stream);
    else if (kind == 1) status = dcg_conv2d_dx(&d, pa, pb, dst, ep.ep, precision, ws.data(), ws.bytes, stream);
    else status = dcg_conv2d_dk(&d, pa, pb, dst, precision, ws.data(), ws.bytes, stream);
    Py_END_ALLOW_THREADS
    check(status);
    if (out == Py_None) return THPVariable_Wrap(std::move(result));
    Py_INCREF(out);
    return out;
}

template <typename F>
PyObject* guarded(Py_ssize_t given, Py_ssize_t wanted, F body)
{
    try {
        if (given != wanted) fail(PyExc_TypeError, "wrong number of arguments");
        return body();
    } catch (const Error&) {
        return nullptr;
    } catch (const c10::OutOfMemoryError& e) {
        PyObject* torch = PyImport_ImportModule("torch");
        PyObject* type = torch ? PyObject_GetAttrString(torch, "OutOfMemoryError") : nullptr;
        if (type) PyErr_SetString(type, e.what_without_backtrace());
        Py_XDECREF(type);
        Py_XDECREF(torch);
    } catch (const c10::Error& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
    }
    return nullptr;
}

// (x, k, strides, pad, out_hw, epilogue, precision, out)
PyObject* conv2d_fwd(PyObject*, PyObject* const* a, Py_ssize_t n)
{
    return guarded(n, 8, [&] {
        const at::Tensor &x = tensor4(a[0]), &k = tensor4(a[1]);
        if (x.size(3) != k.size(2)) fail(PyExc_AssertionError, "kernel input channels differ from activation channels");
        const dcg_conv_desc d = describe((int)x.size(0), (int)x.size(1), (int)x.size(2), (int)x.size(3), (int)k.size(0), (int)k.size(1),
                                         (int)k.size(3), a[2], a[3], a[4]);
        return run_conv(0, d, x, k, a[5], to_int(a[6]), a[7]);
    });
}

// (dy, k, in_hw, strides, pad, epilogue, precision, out)
PyObject* conv2d_dx(PyObject*, PyObject* const* a, Py_ssize_t n)
{
    return guarded(n, 8, [&] {
        const at::Tensor &dy = tensor4(a[0]), &k = tensor4(a[1]);
        if (dy.size(3) != k.size(3)) fail(PyExc_AssertionError, "kernel output channels differ from gradient channels");
        int h, w;
        pair(a[2], h, w);
        dcg_conv_desc d = describe((int)dy.size(0), h, w, (int)k.size(2), (int)k.size(0), (int)k.size(1), (int)k.size(3), a[3], a[4], Py_None);
        d.ho = (int)dy.size(1); d.wo = (int)dy.size(2);
        return run_conv(1, d, dy, k, a[5], to_int(a[6]), a[7]);
    });
}

// (x, dy, k_hw, strides, pad, precision, out)
PyObject* conv2d_dk(PyObject*, PyObject* const* a, Py_ssize_t n)
{
    return guarded(n, 7, [&] {
        const at::Tensor &x = tensor4(a[0]), &dy = tensor4(a[1]);
        if (x.size(0) != dy.size(0)) fail(PyExc_AssertionError, "batch sizes differ");
        int kh, kw;
        pair(a[2], kh, kw);
        dcg_conv_desc d = describe((int)x.size(0), (int)x.size(1), (int)x.size(2), (int)x.size(3), kh, kw, (int)dy.size(3), a[3], a[4], Py_None);
        d.ho = (int)dy.size(1); d.wo = (int)dy.size(2);
        return run_conv(2, d, x, dy, Py_None, to_int(a[5]), a[6]);
    });
}

// (a, out)
PyObject* colsum(PyObject*, PyObject* const* a, Py_ssize_t n)
{
    return guarded(n, 2, [&]() -> PyObject* {
        const at::Tensor& t = tensor(a[0]);
        if (t.dim() == 0 || t.size(t.dim() - 1) == 0) fail(PyExc_ValueError, "colsum: no columns");
        const int64_t cols = t.size(t.dim() - 1), rows = t.numel() / cols;
        at::Tensor result;
        float* dst;
        if (a[1] == Py_None) {
            result = new_tensor({cols}, at::kFloat, t.device());
            dst = static_cast<float*>(result.data_ptr());
        } else {
            dst = static_cast<float*>(tensor(a[1]).data_ptr());
        }
        const Scratch ws(dcg_colsum_workspace_bytes((size_t)rows, (size_t)cols), t.device());
        const float* src = static_cast<const float*>(t.data_ptr());
        void* stream = c10::cuda::getCurrentCUDAStream().stream();
        int status;
        Py_BEGIN_ALLOW_THREADS
        status = dcg_colsum(src, dst, (size_t)rows, (size_t)cols, ws.data(), ws.bytes, stream);
        Py_END_ALLOW_THREADS
        check(status);
        if (a[1] == Py_None) return THPVariable_Wrap(std::move(result));
        Py_INCREF(a[1]);
        return a[1];
    });
}

// (epilogue, raw_out, bias, pre_act, act, alpha, gate, gate_act, gate_alpha): fills a ctypes Epilogue and returns it
PyObject* fill_epilogue(PyObject*, PyObject* const* a, Py_ssize_t n)
{
    return guarded(n, 9, [&] {
        const EpilogueView view(a[0], PyBUF_WRITABLE);
        dcg_epilogue* e = const_cast<dcg_epilogue*>(view.ep);
        if (!e) fail(PyExc_TypeError, "expected an Epilogue");
        e->raw_out = pointer(a[1]); e->bias = pointer(a[2]); e->pre_act = pointer(a[3]);
        e->act = (decltype(e->act))to_int(a[4]); e->alpha = to_float(a[5]);
        e->gate = pointer(a[6]);
        e->gate_act = (decltype(e->gate_act))to_int(a[7]); e->gate_alpha = to_float(a[8]);
        Py_INCREF(a[0]);
        return a[0];
    });
}

// (check, Epilogue): what this module needs of _lib
PyObject* set_up(PyObject*, PyObject* const* a, Py_ssize_t n)
{
    return guarded(n, 2, [&]() -> PyObject* {
        Py_INCREF(a[0]);
        Py_XSETREF(g_check, a[0]);
        Py_INCREF(a[1]);
        Py_XSETREF(g_epilogue, a[1]);
        Py_RETURN_NONE;
    });
}

template <typename F>
PyCFunction fastcall(F f) { return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)); }

PyMethodDef g_methods[] = {
    {"conv2d_fwd", fastcall(conv2d_fwd), METH_FASTCALL, nullptr},
    {"conv2d_dx", fastcall(conv2d_dx), METH_FASTCALL, nullptr},
    {"conv2d_dk", fastcall(conv2d_dk), METH_FASTCALL, nullptr},
    {"colsum", fastcall(colsum), METH_FASTCALL, nullptr},
    {"fill_epilogue", fastcall(fill_epilogue), METH_FASTCALL, nullptr},
    {"set_up", fastcall(set_up), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_binding", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__binding() { return PyModule_Create(&g_module); }
