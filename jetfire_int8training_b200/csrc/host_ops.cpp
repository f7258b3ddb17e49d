// The operators' host path as a CPython module: argument checks, output allocation and the call into the C ABI.
//
// What it is for.  A small operator call (a LayerNorm of [1024 x 256]: 2.6 us on the device) spends its time on the host.  Through ctypes
// and torch's Python functions a call took 16-22 us: ~0.5 us per attribute read or view, ~1.5 us per torch.empty, ~3 us for the ctypes
// conversion of a dozen arguments.  Here a call reads the tensors' fields directly, allocates its outputs in their final shapes from the
// caching allocator and passes pointers on.  The Python functions in Nonlinear/ and Linear/ keep the public signatures and documentation
// and hand their arguments over positionally (METH_FASTCALL: no tuple, no keyword parsing).
//
// Conventions shared by all functions: payloads are any 1-byte dtype (int8, or float8_e4m3fn views of it); tensors that are not
// contiguous are copied; 2-D inputs give 2-D outputs, inputs of higher rank are flattened over the leading dimensions and outputs are
// [shape[0], -1, columns]; everything runs on the current stream of the current device.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <vector>

#include "../../include/jetfire_b200.h"

namespace {

using at::Tensor;

PyObject* g_jetfire_error = nullptr;      // _lib.JetfireError

struct PyError {};                         // a Python exception is set

[[noreturn]] void fail(PyObject* type, const char* msg) {
    PyErr_SetString(type, msg);
    throw PyError{};
}

void check(int status, const char* what) {
    if (status == JF_OK) return;
    char buf[256];
    if (status == JF_ERR_LAUNCH) snprintf(buf, sizeof buf, "%s: %s (cuda error %d)", what, jf_status_string(status), jf_last_cuda_error());
    else snprintf(buf, sizeof buf, "%s: %s", what, jf_status_string(status));
    fail(g_jetfire_error, buf);
}

const Tensor& tensor_arg(PyObject* o) {
    if (!THPVariable_Check(o)) fail(PyExc_TypeError, "a torch.Tensor is expected");
    return THPVariable_Unpack(o);
}
const Tensor& cuda_arg(PyObject* o) {
    const Tensor& t = tensor_arg(o);
    if (!t.is_cuda()) fail(PyExc_RuntimeError, "jetfire_int8training_b200 operators need CUDA tensors (there is no CPU path)");
    return t;
}
int64_t int_arg(PyObject* o) {
    const int64_t v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw PyError{};
    return v;
}
uint64_t u64_arg(PyObject* o) {
    const uint64_t v = PyLong_AsUnsignedLongLongMask(o);
    if (v == (uint64_t)-1 && PyErr_Occurred()) throw PyError{};
    return v;
}
bool bool_arg(PyObject* o) {
    const int v = PyObject_IsTrue(o);
    if (v < 0) throw PyError{};
    return v != 0;
}

void* stream() { return (void*)c10::cuda::getCurrentCUDAStream().stream(); }

// A matrix argument: contiguous storage, flattened to [M, N]
struct Mat {
    Tensor t;
    int64_t M, N, batch;      // batch = shape[0] of an input with rank != 2, else -1
};
Mat mat(const Tensor& x) {
    if (x.dim() < 1) fail(PyExc_RuntimeError, "a matrix is expected");
    Mat m{x.is_contiguous() ? x : x.contiguous(), 0, x.size(-1), -1};
    m.M = m.N > 0 ? x.numel() / m.N : 0;
    if (x.dim() != 2) m.batch = x.size(0);
    return m;
}
Mat payload(PyObject* o) {
    const Tensor& x = cuda_arg(o);
    if (x.element_size() != 1) fail(PyExc_RuntimeError, "an int8 payload is expected");
    return mat(x);
}
Mat floating(PyObject* o, int* dtype) {
    const Tensor& x = cuda_arg(o);
    switch (x.scalar_type()) {
        case at::kFloat: *dtype = JF_F32; return mat(x);
        case at::kHalf: *dtype = JF_F16; return mat(x);
        case at::kBFloat16: *dtype = JF_BF16; return mat(x);
        default: *dtype = JF_F32; return mat(x.to(at::kFloat));
    }
}
Tensor contiguous(const Tensor& t) { return t.is_contiguous() ? t : t.contiguous(); }
Tensor fp32_vector(PyObject* o) {
    const Tensor& t = cuda_arg(o);
    return contiguous(t.scalar_type() == at::kFloat ? t : t.detach().to(at::kFloat));
}

Tensor empty(at::IntArrayRef shape, at::ScalarType dt, const Tensor& like) {
    return at::detail::empty_cuda(shape, dt, like.device(), std::nullopt);
}
// an output of `rows` rows and `cols` columns in the shape convention of an input
Tensor out(const Mat& like, int64_t rows, int64_t cols, at::ScalarType dt) {
    if (like.batch < 0) return empty({rows, cols}, dt, like.t);
    if (like.batch == 0 || rows % like.batch != 0) fail(PyExc_RuntimeError, "the rows of one batch element must be a multiple of 32");
    return empty({like.batch, rows / like.batch, cols}, dt, like.t);
}
Tensor out_scales(const Mat& like) { return out(like, like.M / 32, like.N / 32, at::kHalf); }
// dimensions are checked before outputs are allocated in their shape
void need_blocks(const Mat& m, const char* what) {
    if (m.M <= 0 || m.N <= 0 || m.M % 32 || m.N % 32) check(JF_ERR_SHAPE, what);
}

// stochastic rounding: (flag, noise tensor or None, seed, offset)
struct Sr {
    int on;
    Tensor noise;
    uint64_t seed = 0, offset = 0;
    const float* ptr() const { return noise.defined() ? noise.const_data_ptr<float>() : nullptr; }
};
Sr sr_args(PyObject* const* a, const Mat& like) {
    Sr s;
    s.on = bool_arg(a[0]);
    if (!s.on) return s;
    if (a[1] != Py_None) {
        s.noise = contiguous(tensor_arg(a[1]).reshape({like.M, like.N}).to(like.t.device(), at::kFloat));
    } else {
        s.seed = u64_arg(a[2]);
        s.offset = u64_arg(a[3]);
    }
    return s;
}

PyObject* wrap(Tensor&& t) { return THPVariable_Wrap(std::move(t)); }
template <class... T>
PyObject* tuple(T&&... ts) {
    PyObject* r = PyTuple_New(sizeof...(ts));
    if (!r) throw PyError{};
    Py_ssize_t i = 0;
    (PyTuple_SET_ITEM(r, i++, wrap(std::move(ts))), ...);
    return r;
}

const int8_t* i8(const Mat& m) { return (const int8_t*)m.t.const_data_ptr(); }
int8_t* i8(const Tensor& t) { return (int8_t*)t.mutable_data_ptr(); }

// ------------------------------------------------------------------------------------------------ nonlinear operators
// quantize(x, with_transpose, transpose_2d, stochastic, noise, seed, offset)
PyObject* quantize(PyObject* const* a) {
    int dt;
    const Mat x = floating(a[0], &dt);
    const bool with_t = bool_arg(a[1]);
    const char* what = with_t ? "int8_quantize_transpose" : "int8_quantize";
    need_blocks(x, what);
    const Sr sr = sr_args(a + 3, x);
    Tensor q = out(x, x.M, x.N, at::kChar), s = out_scales(x), qt;
    if (with_t) {
        if (x.batch >= 0 && !bool_arg(a[2])) {
            if (x.N % x.batch) fail(PyExc_RuntimeError, "the transposed copy cannot be split over the batch");
            qt = empty({x.batch, x.N / x.batch, x.M}, at::kChar, x.t);
        } else {
            qt = empty({x.N, x.M}, at::kChar, x.t);
        }
    }
    check(jf_int8_quantize(x.t.const_data_ptr(), dt, x.M, x.N, i8(q), s.mutable_data_ptr(), with_t ? i8(qt) : nullptr, sr.on, sr.ptr(), sr.seed,
                           sr.offset, stream()), what);
    return with_t ? tuple(std::move(q), std::move(s), std::move(qt)) : tuple(std::move(q), std::move(s));
}

// quantize_many(sequence of 2-D tensors of one dtype and device): one launch per eight tensors
PyObject* quantize_many(PyObject* const* a) {
    PyObject* seq = PySequence_Fast(a[0], "a sequence of tensors is expected");
    if (!seq) throw PyError{};
    struct Guard { PyObject* o; ~Guard() { Py_DECREF(o); } } guard{seq};
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(seq);
    std::vector<Mat> x;
    x.reserve(n);
    int dt = JF_F32;
    for (Py_ssize_t i = 0; i < n; ++i) {
        int d;
        x.push_back(floating(PySequence_Fast_GET_ITEM(seq, i), &d));
        if (i > 0 && d != dt) fail(PyExc_AssertionError, "int8_quantize_many: the tensors have different dtypes");
        dt = d;
        if (x[i].batch >= 0 || x[i].t.device() != x[0].t.device()) fail(PyExc_AssertionError, "int8_quantize_many: 2-D tensors of one device are expected");
        need_blocks(x[i], "int8_quantize_many");
    }
    PyObject* list = PyList_New(n);
    if (!list) throw PyError{};
    struct ListGuard { PyObject* o; ~ListGuard() { Py_XDECREF(o); } } list_guard{list};
    for (Py_ssize_t i = 0; i < n; i += 8) {
        const int m = (int)std::min<Py_ssize_t>(8, n - i);
        const void* xp[8]; int64_t M[8], N[8]; int8_t* qp[8]; void* sp[8];
        for (int j = 0; j < m; ++j) {
            const Mat& v = x[i + j];
            Tensor q = out(v, v.M, v.N, at::kChar), sc = out_scales(v);
            xp[j] = v.t.const_data_ptr(); M[j] = v.M; N[j] = v.N; qp[j] = i8(q); sp[j] = sc.mutable_data_ptr();
            PyList_SET_ITEM(list, i + j, tuple(std::move(q), std::move(sc)));
        }
        check(jf_int8_quantize_multi(m, xp, dt, M, N, qp, sp, stream()), "int8_quantize_many");
    }
    list_guard.o = nullptr;
    return list;
}

// transpose(x, transpose_2d)
PyObject* transpose(PyObject* const* a) {
    const Mat x = payload(a[0]);
    need_blocks(x, "int8_transpose");
    Tensor y;
    if (x.batch >= 0 && !bool_arg(a[1])) {
        if (x.N % x.batch) fail(PyExc_RuntimeError, "the transposed copy cannot be split over the batch");
        y = empty({x.batch, x.N / x.batch, x.M}, at::kChar, x.t);
    } else {
        y = empty({x.N, x.M}, at::kChar, x.t);
    }
    check(jf_int8_transpose(i8(x), x.M, x.N, i8(y), stream()), "int8_transpose");
    return wrap(std::move(y));
}

// dequantize(x, s_x)
PyObject* dequantize(PyObject* const* a) {
    const Mat x = payload(a[0]);
    const Tensor s = contiguous(cuda_arg(a[1]));
    need_blocks(x, "int8_dequantize");
    Tensor y = out(x, x.M, x.N, at::kFloat);
    check(jf_int8_dequantize(i8(x), s.const_data_ptr(), x.M, x.N, y.mutable_data_ptr<float>(), stream()), "int8_dequantize");
    return wrap(std::move(y));
}

// gelu_forward(x, s_x)
PyObject* gelu_forward(PyObject* const* a) {
    const Mat x = payload(a[0]);
    const Tensor s = contiguous(cuda_arg(a[1]));
    need_blocks(x, "int8_gelu_forward");
    Tensor y = out(x, x.M, x.N, at::kChar), sy = out_scales(x);
    check(jf_int8_gelu_forward(i8(x), s.const_data_ptr(), x.M, x.N, i8(y), sy.mutable_data_ptr(), stream()), "int8_gelu_forward");
    return tuple(std::move(y), std::move(sy));
}

// gelu_backward(x, s_x, g, s_g, stochastic, noise, seed, offset)
PyObject* gelu_backward(PyObject* const* a) {
    const Mat x = payload(a[0]), g = payload(a[2]);
    const Tensor sx = contiguous(cuda_arg(a[1])), sg = contiguous(cuda_arg(a[3]));
    need_blocks(x, "int8_gelu_backward");
    const Sr sr = sr_args(a + 4, x);
    Tensor y = out(x, x.M, x.N, at::kChar), sy = out_scales(x);
    check(jf_int8_gelu_backward(i8(x), sx.const_data_ptr(), i8(g), sg.const_data_ptr(), x.M, x.N, i8(y), sy.mutable_data_ptr(), sr.on, sr.ptr(),
                                sr.seed, sr.offset, stream()), "int8_gelu_backward");
    return tuple(std::move(y), std::move(sy));
}

// layernorm_forward(x, sx, weight, mean, rstd)
PyObject* layernorm_forward(PyObject* const* a) {
    const Mat x = payload(a[0]);
    const Tensor s = contiguous(cuda_arg(a[1])), w = fp32_vector(a[2]), mu = fp32_vector(a[3]), rs = fp32_vector(a[4]);
    need_blocks(x, "int8_layernorm_forward");
    Tensor y = out(x, x.M, x.N, at::kChar), sy = out_scales(x);
    check(jf_int8_layernorm_forward(i8(x), s.const_data_ptr(), w.const_data_ptr<float>(), mu.const_data_ptr<float>(), rs.const_data_ptr<float>(),
                                    x.M, x.N, i8(y), sy.mutable_data_ptr(), stream()), "int8_layernorm_forward");
    return tuple(std::move(y), std::move(sy));
}

// layernorm_backward(x, sx, g, sg, w, mean, rstd, stochastic, noise, seed, offset)
PyObject* layernorm_backward(PyObject* const* a) {
    const Mat x = payload(a[0]), g = payload(a[2]);
    const Tensor sx = contiguous(cuda_arg(a[1])), sg = contiguous(cuda_arg(a[3]));
    const at::ScalarType w_type = cuda_arg(a[4]).scalar_type();
    const Tensor w = fp32_vector(a[4]), mu = fp32_vector(a[5]), rs = fp32_vector(a[6]);
    need_blocks(x, "int8_layernorm_backward");
    const Sr sr = sr_args(a + 7, x);
    Tensor dx = out(x, x.M, x.N, at::kChar), sdx = out_scales(x), dw = empty({x.N}, at::kFloat, x.t);
    const Tensor scratch = empty({(x.M / 32) * x.N}, at::kFloat, x.t);
    check(jf_int8_layernorm_backward(i8(x), sx.const_data_ptr(), i8(g), sg.const_data_ptr(), w.const_data_ptr<float>(), mu.const_data_ptr<float>(),
                                     rs.const_data_ptr<float>(), x.M, x.N, 128, i8(dx), sdx.mutable_data_ptr(), dw.mutable_data_ptr<float>(),
                                     scratch.mutable_data_ptr<float>(), sr.on, sr.ptr(), sr.seed, sr.offset, stream()),
          "int8_layernorm_backward");
    if (w_type != at::kFloat) dw = dw.to(w_type);
    return tuple(std::move(dx), std::move(sdx), std::move(dw));
}

// add(x1, x2, s_x2, mean_var, stochastic, noise, seed, offset)
PyObject* add(PyObject* const* a) {
    int dt;
    const Mat x = floating(a[0], &dt), q = payload(a[1]);
    const Tensor s = contiguous(cuda_arg(a[2]));
    const bool mean_var = bool_arg(a[3]);
    const char* what = mean_var ? "int8_add_Ifp_Ig16_Ofp_Og_MeanVar" : "int8_add_Ifp_Ig16_Ofp_Og";
    if (x.M != q.M || x.N != q.N) fail(PyExc_AssertionError, "the two addends have different shapes");
    need_blocks(x, what);
    const Sr sr = sr_args(a + 4, x);
    Tensor y = out(x, x.M, x.N, at::kFloat), y2 = out(x, x.M, x.N, at::kChar), sy = out_scales(x);
    if (!mean_var) {
        check(jf_int8_add(x.t.const_data_ptr(), dt, i8(q), s.const_data_ptr(), x.M, x.N, y.mutable_data_ptr<float>(), i8(y2), sy.mutable_data_ptr(),
                          sr.on, sr.ptr(), sr.seed, sr.offset, stream()), what);
        return tuple(std::move(y), std::move(y2), std::move(sy));
    }
    Tensor mean = x.batch < 0 ? empty({x.M}, at::kFloat, x.t) : empty({x.batch, x.M / x.batch}, at::kFloat, x.t);
    Tensor rstd = x.batch < 0 ? empty({x.M}, at::kFloat, x.t) : empty({x.batch, x.M / x.batch}, at::kFloat, x.t);
    const Tensor scratch = empty({2 * x.M * ((x.N + 127) / 128)}, at::kFloat, x.t);
    check(jf_int8_add_meanvar(x.t.const_data_ptr(), dt, i8(q), s.const_data_ptr(), x.M, x.N, y.mutable_data_ptr<float>(), i8(y2),
                              sy.mutable_data_ptr(), mean.mutable_data_ptr<float>(), rstd.mutable_data_ptr<float>(),
                              scratch.mutable_data_ptr<float>(), stream()), what);
    return tuple(std::move(y), std::move(y2), std::move(sy), std::move(mean), std::move(rstd));
}

// ------------------------------------------------------------------------------------------------ linear layer
// A scale argument of a linear operator: [rows/32, columns/32] after flattening
struct Scale {
    Tensor t;
    int64_t cols;
};
Scale scale_arg(PyObject* o) {
    const Tensor& t = cuda_arg(o);
    return Scale{contiguous(t), t.size(-1)};
}
// leading dimensions of `like` (before any flattening) with another last dimension
Tensor out_last(const Tensor& like, int64_t last, at::ScalarType dt) {
    c10::SmallVector<int64_t, 6> shape(like.sizes().begin(), like.sizes().end());
    shape.back() = last;
    return empty(shape, dt, like);
}

// linear_forward(x, sx, w, sw, output_quantized)
PyObject* linear_forward(PyObject* const* a) {
    const Mat x = payload(a[0]), w = payload(a[2]);
    const Tensor& sx_in = cuda_arg(a[1]);
    const Scale sx = scale_arg(a[1]), sw = scale_arg(a[3]);
    const int64_t M = x.M, K = x.N, N = w.t.size(0);
    const char* what = "int8_linear_forward";
    if (M <= 0 || M % 32 || K % 32 || N <= 0 || N % 32) check(JF_ERR_SHAPE, what);
    const bool quantised = bool_arg(a[4]);
    Tensor y = out_last(tensor_arg(a[0]), N, quantised ? at::kChar : at::kHalf);
    Tensor sy = quantised ? out_last(sx_in, N / 32, at::kHalf) : Tensor();
    if (quantised && sy.numel() != (M / 32) * (N / 32)) fail(PyExc_RuntimeError, "the scales do not fit the payload");
    check(jf_igemm_forward(i8(x), i8(w), sx.t.const_data_ptr(), sx.cols, 1, sw.t.const_data_ptr(), sw.cols, 1, M, N, K,
                           quantised ? JF_OUT_INT8 : JF_OUT_DEQUANT_F16, quantised ? i8(y) : nullptr, quantised ? sy.mutable_data_ptr() : nullptr,
                           quantised ? nullptr : y.mutable_data_ptr(), nullptr, 0, stream()), what);
    return quantised ? tuple(std::move(y), std::move(sy)) : wrap(std::move(y));
}

Tensor wgrad(const Mat& x, const Scale& sx, const Mat& g, const Scale& sg, at::ScalarType dt, int split_k) {
    const int64_t T = g.M, cout = g.N, cin = x.N;
    const int splits = jf_igemm_wgrad_plan(cout, cin, T, split_k);
    if (splits < 1) check(splits, "int8_linear_wgrad(plan)");
    Tensor dw = empty({cout, cin}, dt, g.t), scratch;
    if (splits > 1) scratch = empty({splits * cout * cin}, at::kFloat, g.t);
    check(jf_igemm_wgrad(i8(g), 0, i8(x), sg.t.const_data_ptr(), sg.cols, 1, sx.t.const_data_ptr(), sx.cols, 1, cout, cin, T,
                         dt == at::kHalf ? JF_F16 : JF_F32, dw.mutable_data_ptr(), splits, splits > 1 ? scratch.mutable_data_ptr<float>() : nullptr,
                         nullptr, 0, stream()), "int8_linear_wgrad");
    return dw;
}

// linear_wgrad(x, sx, g, sg, fp16, split_k)
PyObject* linear_wgrad(PyObject* const* a) {
    const Mat x = payload(a[0]), g = payload(a[2]);
    return wrap(wgrad(x, scale_arg(a[1]), g, scale_arg(a[3]), bool_arg(a[4]) ? at::kHalf : at::kFloat, (int)int_arg(a[5])));
}

// linear_backward(x, sx, g, sg, w, sw, quantised, wgrad_fp16, split_k, stochastic, noise, seed, offset)
PyObject* linear_backward(PyObject* const* a) {
    const Mat x = payload(a[0]), g = payload(a[2]), w = payload(a[4]);
    const Tensor& sg_in = cuda_arg(a[3]);
    const Scale sx = scale_arg(a[1]), sg = scale_arg(a[3]), sw = scale_arg(a[5]);
    const int64_t cout = w.t.size(0), cin = w.N, M = g.M;
    const char* what = "int8_linear_backward(dgrad)";
    if (M <= 0 || M % 32 || cin <= 0 || cin % 32 || cout <= 0 || cout % 32) check(JF_ERR_SHAPE, what);
    if (g.N != cout || x.N != cin) fail(PyExc_RuntimeError, "int8_linear_backward: the last dimensions do not fit the weight");
    const bool quantised = bool_arg(a[6]);
    const Mat like{g.t, M, cin, -1};
    const Sr sr = sr_args(a + 9, like);
    Tensor gx = out_last(tensor_arg(a[2]), cin, quantised ? at::kChar : at::kHalf);
    Tensor gsx = quantised ? out_last(sg_in, cin / 32, at::kHalf) : Tensor();
    if (quantised && gsx.numel() != (M / 32) * (cin / 32)) fail(PyExc_RuntimeError, "the scales do not fit the payload");
    check(jf_igemm_dgrad(i8(g), i8(w), sg.t.const_data_ptr(), sg.cols, 1, sw.t.const_data_ptr(), sw.cols, 1, M, cin, cout,
                         quantised ? JF_OUT_INT8 : JF_OUT_DEQUANT_F16, quantised ? i8(gx) : nullptr, quantised ? gsx.mutable_data_ptr() : nullptr,
                         quantised ? nullptr : gx.mutable_data_ptr(), sr.on, sr.ptr(), sr.seed, sr.offset, nullptr, 0, stream()), what);
    Tensor gw = wgrad(x, sx, g, sg, bool_arg(a[7]) ? at::kHalf : at::kFloat, (int)int_arg(a[8]));
    return quantised ? tuple(std::move(gx), std::move(gsx), std::move(gw)) : tuple(std::move(gx), std::move(gw));
}

// ------------------------------------------------------------------------------------------------ module
template <PyObject* (*F)(PyObject* const*), int N>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != N) {
        PyErr_Format(PyExc_TypeError, "%d arguments are expected", N);
        return nullptr;
    }
    try {
        return F(args);
    } catch (const PyError&) {
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
}

PyObject* set_error_class(PyObject*, PyObject* cls) {
    Py_INCREF(cls);
    Py_XDECREF(g_jetfire_error);
    g_jetfire_error = cls;
    Py_RETURN_NONE;
}

#define JF_ENTRY(name, n) {#name, (PyCFunction)(void (*)(void))entry<name, n>, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    JF_ENTRY(quantize, 7), JF_ENTRY(quantize_many, 1), JF_ENTRY(transpose, 2), JF_ENTRY(dequantize, 2), JF_ENTRY(gelu_forward, 2), JF_ENTRY(gelu_backward, 8),
    JF_ENTRY(layernorm_forward, 5), JF_ENTRY(layernorm_backward, 11), JF_ENTRY(add, 8), JF_ENTRY(linear_forward, 5),
    JF_ENTRY(linear_wgrad, 6), JF_ENTRY(linear_backward, 13), {"set_error_class", set_error_class, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host_ops", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host_ops(void) { return PyModule_Create(&module); }
