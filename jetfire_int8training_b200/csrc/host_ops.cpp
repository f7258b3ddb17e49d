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
#include <ATen/core/LegacyTypeDispatch.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <array>
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
    int64_t M = 0, N = 0, batch = -1;      // batch = shape[0] of an input with rank != 2, else -1
};
Mat mat(const Tensor& x) {
    if (x.dim() < 1) fail(PyExc_RuntimeError, "a matrix is expected");
    Mat m;
    m.t = x.is_contiguous() ? x : x.contiguous();
    m.N = x.size(-1);
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

// quantize_parts(parts, stochastic, noise (None), seed, offset): the parts are [..., cols] tensors of one shape and dtype
PyObject* quantize_parts(PyObject* const* a) {
    PyObject* seq = PySequence_Fast(a[0], "a sequence of tensors is expected");
    if (!seq) throw PyError{};
    struct Guard { PyObject* o; ~Guard() { Py_DECREF(o); } } guard{seq};
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(seq);
    if (n < 1 || n > 4) fail(PyExc_ValueError, "int8_quantize_parts takes one to four parts");
    Mat x[4];
    const void* p[4];
    int dt = JF_F32;
    for (Py_ssize_t i = 0; i < n; ++i) {
        int d;
        x[i] = floating(PySequence_Fast_GET_ITEM(seq, i), &d);
        if (i > 0 && (d != dt || x[i].M != x[0].M || x[i].N != x[0].N)) fail(PyExc_ValueError, "int8_quantize_parts: parts of one shape and dtype are expected");
        dt = d;
        p[i] = x[i].t.const_data_ptr();
    }
    Mat whole = x[0];
    whole.N *= n;
    need_blocks(x[0], "int8_quantize_parts");
    const Sr sr = sr_args(a + 1, whole);
    if (sr.noise.defined()) fail(PyExc_ValueError, "int8_quantize_parts generates its noise");
    Tensor q = out(whole, whole.M, whole.N, at::kChar), sc = out_scales(whole);
    check(jf_int8_quantize_parts((int)n, p, dt, whole.M, x[0].N, i8(q), sc.mutable_data_ptr(), sr.on, sr.seed, sr.offset, stream()), "int8_quantize_parts");
    return tuple(std::move(q), std::move(sc));
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

// add(x1, x2, s_x2, mean_var, bf16_out, stochastic, noise, seed, offset)
PyObject* add(PyObject* const* a) {
    int dt;
    const Mat x = floating(a[0], &dt), q = payload(a[1]);
    const Tensor s = contiguous(cuda_arg(a[2]));
    const bool mean_var = bool_arg(a[3]);
    const char* what = mean_var ? "int8_add_Ifp_Ig16_Ofp_Og_MeanVar" : "int8_add_Ifp_Ig16_Ofp_Og";
    if (x.M != q.M || x.N != q.N) fail(PyExc_AssertionError, "the two addends have different shapes");
    need_blocks(x, what);
    const bool narrow = bool_arg(a[4]);
    const int ydt = narrow ? JF_BF16 : JF_F32;
    const Sr sr = sr_args(a + 5, x);
    Tensor y = out(x, x.M, x.N, narrow ? at::kBFloat16 : at::kFloat), y2 = out(x, x.M, x.N, at::kChar), sy = out_scales(x);
    if (!mean_var) {
        check(jf_int8_add_out(x.t.const_data_ptr(), dt, i8(q), s.const_data_ptr(), x.M, x.N, y.mutable_data_ptr(), ydt, i8(y2), sy.mutable_data_ptr(),
                          sr.on, sr.ptr(), sr.seed, sr.offset, stream()), what);
        return tuple(std::move(y), std::move(y2), std::move(sy));
    }
    Tensor mean = x.batch < 0 ? empty({x.M}, at::kFloat, x.t) : empty({x.batch, x.M / x.batch}, at::kFloat, x.t);
    Tensor rstd = x.batch < 0 ? empty({x.M}, at::kFloat, x.t) : empty({x.batch, x.M / x.batch}, at::kFloat, x.t);
    const Tensor scratch = empty({2 * x.M * ((x.N + 127) / 128)}, at::kFloat, x.t);
    check(jf_int8_add_meanvar_out(x.t.const_data_ptr(), dt, i8(q), s.const_data_ptr(), x.M, x.N, y.mutable_data_ptr(), ydt, i8(y2),
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

// dW and the workspace of its split sum
struct Wgrad {
    Tensor dw, scratch;
    int dtype, splits;
    Wgrad(const Mat& x, const Mat& g, bool fp16, int split_k) : dtype(fp16 ? JF_F16 : JF_F32) {
        const int64_t cout = g.N, cin = x.N;
        splits = jf_igemm_wgrad_plan(cout, cin, g.M, split_k);
        if (splits < 1) check(splits, "int8_linear_wgrad(plan)");
        dw = empty({cout, cin}, fp16 ? at::kHalf : at::kFloat, g.t);
        if (splits > 1) scratch = empty({splits * cout * cin}, at::kFloat, g.t);
    }
    float* workspace() const { return splits > 1 ? scratch.mutable_data_ptr<float>() : nullptr; }
};

// linear_wgrad(x, sx, g, sg, fp16, split_k)
PyObject* linear_wgrad(PyObject* const* a) {
    const Mat x = payload(a[0]), g = payload(a[2]);
    const Scale sx = scale_arg(a[1]), sg = scale_arg(a[3]);
    Wgrad w(x, g, bool_arg(a[4]), (int)int_arg(a[5]));
    check(jf_igemm_wgrad(i8(g), 0, i8(x), sg.t.const_data_ptr(), sg.cols, 1, sx.t.const_data_ptr(), sx.cols, 1, g.N, x.N, g.M, w.dtype,
                         w.dw.mutable_data_ptr(), w.splits, w.workspace(), nullptr, 0, stream()), "int8_linear_wgrad");
    return wrap(std::move(w.dw));
}

// linear_backward(x, sx, g, sg, w, sw, quantised, wgrad_fp16, split_k, stochastic, noise, seed, offset)
PyObject* linear_backward(PyObject* const* a) {
    const Mat x = payload(a[0]), g = payload(a[2]), w = payload(a[4]);
    const Tensor& sg_in = cuda_arg(a[3]);
    const Scale sx = scale_arg(a[1]), sg = scale_arg(a[3]), sw = scale_arg(a[5]);
    const int64_t cout = w.t.size(0), cin = w.N, M = g.M;
    const char* what = "int8_linear_backward";
    if (M <= 0 || M % 32 || cin <= 0 || cin % 32 || cout <= 0 || cout % 32) check(JF_ERR_SHAPE, what);
    if (g.N != cout || x.N != cin) fail(PyExc_RuntimeError, "int8_linear_backward: the last dimensions do not fit the weight");
    const bool quantised = bool_arg(a[6]);
    Mat like;
    like.t = g.t; like.M = M; like.N = cin;
    const Sr sr = sr_args(a + 9, like);
    Tensor gx = out_last(tensor_arg(a[2]), cin, quantised ? at::kChar : at::kHalf);
    Tensor gsx = quantised ? out_last(sg_in, cin / 32, at::kHalf) : Tensor();
    if (quantised && gsx.numel() != (M / 32) * (cin / 32)) fail(PyExc_RuntimeError, "the scales do not fit the payload");
    Wgrad dw(x, g, bool_arg(a[7]), (int)int_arg(a[8]));
    check(jf_igemm_backward(i8(g), i8(w), i8(x), sg.t.const_data_ptr(), sg.cols, 1, sw.t.const_data_ptr(), sw.cols, 1, sx.t.const_data_ptr(),
                            sx.cols, 1, M, cout, cin, quantised ? JF_OUT_INT8 : JF_OUT_DEQUANT_F16, quantised ? i8(gx) : nullptr,
                            quantised ? gsx.mutable_data_ptr() : nullptr, quantised ? nullptr : gx.mutable_data_ptr(), sr.on, sr.ptr(),
                            sr.seed, sr.offset, dw.dtype, dw.dw.mutable_data_ptr(), dw.splits, dw.workspace(), stream()), what);
    return quantised ? tuple(std::move(gx), std::move(gsx), std::move(dw.dw)) : tuple(std::move(gx), std::move(dw.dw));
}

// ------------------------------------------------------------------------------------------------ the GPT-2 caller's floating-point parts
struct NoGil {
    PyThreadState* state = PyEval_SaveThread();
    ~NoGil() { PyEval_RestoreThread(state); }
};
// framework operators called from inside an autograd Function: no graph, no autocast
struct Plain {
    at::AutoDispatchBelowADInplaceOrView below;
    c10::impl::ExcludeDispatchKeyGuard no_autocast{c10::autocast_dispatch_keyset};
};

PyObject* wrap_or_none(const Tensor& t) {
    if (!t.defined()) Py_RETURN_NONE;
    return THPVariable_Wrap(t);
}
Tensor tensor_or_undefined(PyObject* o) { return o == Py_None ? Tensor() : tensor_arg(o); }

// [B, T, 3C] -> q, k, v as [B, heads, T, C / heads] views
std::array<Tensor, 3> split_heads(const Tensor& qkv, int64_t heads) {
    const int64_t B = qkv.size(0), T = qkv.size(1), C = qkv.size(2) / 3, hs = C / heads;
    const auto st = qkv.strides();
    std::array<Tensor, 3> r;
    for (int i = 0; i < 3; ++i)
        r[i] = qkv.as_strided({B, heads, T, hs}, {st[0], hs * st[2], st[1], st[2]}, qkv.storage_offset() + i * C * st[2]);
    return r;
}
// [B, heads, T, hs] -> [B, T, C], without a copy when the memory is laid out that way
Tensor join_heads(const Tensor& t) { return t.transpose(1, 2).contiguous().view({t.size(0), t.size(2), t.size(1) * t.size(3)}); }

// attention_forward(qkv [B, T, 3C], heads): causal attention through the fused operator that scaled_dot_product_attention would pick, or None
// when that is not the cuDNN one.  -> (y [B, T, C], max_q, max_k, out, logsumexp, philox_seed, philox_offset, cum_seq_q, cum_seq_k)
PyObject* attention_forward(PyObject* const* a) {
    const Tensor& qkv = cuda_arg(a[0]);
    const int64_t heads = int_arg(a[1]);
    if (qkv.dim() != 3 || qkv.size(2) % (3 * heads)) fail(PyExc_RuntimeError, "attention_forward: [B, T, 3C] is expected");
    Tensor y;
    std::tuple<Tensor, Tensor, Tensor, Tensor, c10::SymInt, c10::SymInt, Tensor, Tensor, Tensor> r;
    {
        NoGil no_gil;
        Plain plain;
        const auto q = split_heads(qkv.detach(), heads);
        int64_t choice;
        {
            c10::AutoGradMode grad(true);       // the choice is the one for inputs that need gradients
            for (auto& t : q) t.set_requires_grad(true);
            choice = at::_fused_sdp_choice(q[0], q[1], q[2], std::nullopt, 0.0, true);
        }
        if (choice == 3 /* cuDNN */) {
            for (auto& t : q) t.set_requires_grad(false);
            r = at::_scaled_dot_product_cudnn_attention(q[0], q[1], q[2], std::nullopt, true, 0.0, true, false);
            y = join_heads(std::get<0>(r));
        }
    }
    if (!y.defined()) Py_RETURN_NONE;
    return Py_BuildValue("(NLLNNNNNN)", wrap(std::move(y)), (long long)std::get<4>(r).guard_int(__FILE__, __LINE__),
                         (long long)std::get<5>(r).guard_int(__FILE__, __LINE__), wrap_or_none(std::get<0>(r)), wrap_or_none(std::get<1>(r)),
                         wrap_or_none(std::get<6>(r)), wrap_or_none(std::get<7>(r)), wrap_or_none(std::get<2>(r)), wrap_or_none(std::get<3>(r)));
}

// attention_backward(gy [B, T, C], qkv, heads, max_q, max_k, out, logsumexp, philox_seed, philox_offset, cum_seq_q, cum_seq_k)
// -> gradients of q, k, v, each [B, T, C]
PyObject* attention_backward(PyObject* const* a) {
    const Tensor &gy = cuda_arg(a[0]), &qkv = cuda_arg(a[1]);
    const int64_t heads = int_arg(a[2]), max_q = int_arg(a[3]), max_k = int_arg(a[4]);
    const Tensor out = tensor_arg(a[5]), lse = tensor_arg(a[6]), seed = tensor_or_undefined(a[7]), offset = tensor_or_undefined(a[8]),
                 cq = tensor_or_undefined(a[9]), ck = tensor_or_undefined(a[10]);
    std::tuple<Tensor, Tensor, Tensor> r;
    Tensor g[3];
    {
        NoGil no_gil;
        Plain plain;
        const auto q = split_heads(qkv.detach(), heads);
        const int64_t B = gy.size(0), T = gy.size(1), C = gy.size(2);
        const Tensor go = gy.detach().reshape({B, T, heads, C / heads}).transpose(1, 2);
        r = at::_scaled_dot_product_cudnn_attention_backward(go, q[0], q[1], q[2], out, lse, seed, offset, Tensor(), cq, ck, max_q, max_k, 0.0, true);
        g[0] = join_heads(std::get<0>(r)); g[1] = join_heads(std::get<1>(r)); g[2] = join_heads(std::get<2>(r));
    }
    return tuple(std::move(g[0]), std::move(g[1]), std::move(g[2]));
}

// The un-quantised ends of the model stay the framework's operators, called without a graph: their last bits decide stochastic roundings
// further down (a differing bit grows to percents of the gradients within a step), so they are not replaced by kernels with another order
// of summation.
// embed_forward(idx [B, T], wte [V, C], wpe [P, C]) -> (x [B, T, C], mean [B, T], rstd [B, T])
PyObject* embed_forward(PyObject* const* a) {
    const Tensor &idx = cuda_arg(a[0]), &wte = cuda_arg(a[1]), &wpe = cuda_arg(a[2]);
    if (idx.dim() != 2 || wpe.dim() != 2 || idx.size(1) > wpe.size(0)) fail(PyExc_ValueError, "embed_forward: idx [B, T] and wpe [P, C] with T <= P are expected");
    Tensor x, mean, rstd;
    {
        NoGil no_gil;
        Plain plain;
        x = at::embedding(wte.detach(), idx);
        x.add_(wpe.detach().slice(0, 0, idx.size(1)));
        mean = x.mean(-1);
        rstd = x.var(-1).sqrt_().reciprocal_();
    }
    return tuple(std::move(x), std::move(mean), std::move(rstd));
}

// embed_backward(idx, g [B, T, C] fp32, head or None, V, P) -> (dwte, dwpe); `head` is the LM head's bf16 gradient of the same matrix, added
// without widening it first
PyObject* embed_backward(PyObject* const* a) {
    const Tensor &idx = cuda_arg(a[0]), &g = cuda_arg(a[1]);
    const Tensor head = tensor_or_undefined(a[2]);
    const int64_t V = int_arg(a[3]), P = int_arg(a[4]);
    Tensor dwte, dwpe;
    int added = JF_OK;
    {
        NoGil no_gil;
        Plain plain;
        dwte = at::embedding_dense_backward(g, idx, V, -1, false);
        if (head.defined() && (dwte.numel() % 8 || !dwte.is_contiguous() || !head.is_contiguous() || head.scalar_type() != at::kBFloat16)) dwte.add_(head);
        else if (head.defined()) added = jf_add_widened(dwte.mutable_data_ptr<float>(), head.const_data_ptr(), dwte.numel(), stream());
        dwpe = g.sum(0);
        if (idx.size(1) < P) {
            Tensor all = at::zeros({P, g.size(2)}, g.options());
            all.slice(0, 0, idx.size(1)).copy_(dwpe);
            dwpe = all;
        }
    }
    check(added, "embed_backward");
    return tuple(std::move(dwte), std::move(dwpe));
}

// final_norm_forward(x [..., C], gamma, eps) -> (y bf16, x fp32, mean, rstd)
PyObject* final_norm_forward(PyObject* const* a) {
    const Tensor &x = cuda_arg(a[0]), &w = cuda_arg(a[1]);
    const double eps = PyFloat_AsDouble(a[2]);
    if (eps == -1.0 && PyErr_Occurred()) throw PyError{};
    Tensor xf, y, mean, rstd;
    {
        NoGil no_gil;
        Plain plain;
        xf = x.detach().to(at::kFloat);
        std::tie(y, mean, rstd) = at::native_layer_norm(xf, {x.size(-1)}, w.detach(), std::nullopt, eps);
        y = y.to(at::kBFloat16);
    }
    return tuple(std::move(y), std::move(xf), std::move(mean), std::move(rstd));
}
// final_norm_backward(dy bf16, x fp32, gamma, mean, rstd, narrow) -> (dx as bf16 or fp32, dgamma)
PyObject* final_norm_backward(PyObject* const* a) {
    const Tensor &dy = cuda_arg(a[0]), &x = cuda_arg(a[1]), &w = cuda_arg(a[2]), &mean = cuda_arg(a[3]), &rstd = cuda_arg(a[4]);
    const bool narrow = bool_arg(a[5]);
    Tensor dx, dw, db;
    {
        NoGil no_gil;
        Plain plain;
        std::tie(dx, dw, db) = at::native_layer_norm_backward(dy.to(at::kFloat), x, {x.size(-1)}, mean, rstd, w.detach(), std::nullopt, {true, true, false});
        if (narrow) dx = dx.to(at::kBFloat16);
    }
    return tuple(std::move(dx), std::move(dw));
}

// lm_loss_forward(logits bf16 [..., V], targets) -> (loss [], logits [rows, V], targets int64 [rows], lse, count [])
PyObject* lm_loss_forward(PyObject* const* a) {
    const Tensor& in = cuda_arg(a[0]);
    if (in.scalar_type() != at::kBFloat16) fail(PyExc_TypeError, "lm_cross_entropy takes bf16 logits");
    const int64_t V = in.size(-1), rows = in.numel() / V;
    Tensor x = contiguous(in.detach()).view({rows, V});
    Tensor t = cuda_arg(a[1]).detach().reshape({-1});
    if (t.scalar_type() != at::kLong) t = t.to(at::kLong);
    t = contiguous(t);
    if (t.numel() != rows) fail(PyExc_RuntimeError, "lm_cross_entropy: one target per row of logits is expected");
    Tensor lse = empty({rows}, at::kFloat, x), loss = empty({}, at::kFloat, x), count = empty({}, at::kFloat, x);
    const Tensor loss_rows = empty({rows}, at::kFloat, x);
    check(jf_lm_loss_forward_mean(x.const_data_ptr(), t.const_data_ptr<int64_t>(), rows, V, lse.mutable_data_ptr<float>(),
                                  loss_rows.mutable_data_ptr<float>(), loss.mutable_data_ptr<float>(), count.mutable_data_ptr<float>(), stream()),
          "lm_cross_entropy");
    return tuple(std::move(loss), std::move(x), std::move(t), std::move(lse), std::move(count));
}
// lm_loss_backward(grad, logits [rows, V], targets, lse, count): the logits become their gradient
PyObject* lm_loss_backward(PyObject* const* a) {
    const Tensor g = fp32_vector(a[0]);
    const Tensor &x = cuda_arg(a[1]), &t = cuda_arg(a[2]), &lse = cuda_arg(a[3]), &count = cuda_arg(a[4]);
    check(jf_lm_loss_backward_mean(x.mutable_data_ptr(), t.const_data_ptr<int64_t>(), lse.const_data_ptr<float>(), g.const_data_ptr<float>(),
                                   count.const_data_ptr<float>(), x.size(0), x.size(1), stream()), "lm_cross_entropy(backward)");
    Py_RETURN_NONE;
}

// gradient_pointers(params): addresses of the parameters' fp32 gradients as packed 64-bit integers (bytes); a gradient of another type or
// layout is replaced by an fp32 contiguous copy
PyObject* gradient_pointers(PyObject* const* a) {
    PyObject* seq = PySequence_Fast(a[0], "a sequence of parameters is expected");
    if (!seq) throw PyError{};
    struct Guard { PyObject* o; ~Guard() { Py_DECREF(o); } } guard{seq};
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(seq);
    PyObject* bytes = PyBytes_FromStringAndSize(nullptr, n * 8);
    if (!bytes) throw PyError{};
    struct BytesGuard { PyObject* o; ~BytesGuard() { Py_XDECREF(o); } } bytes_guard{bytes};
    uint64_t* p = reinterpret_cast<uint64_t*>(PyBytes_AS_STRING(bytes));
    for (Py_ssize_t i = 0; i < n; ++i) {
        const Tensor& t = tensor_arg(PySequence_Fast_GET_ITEM(seq, i));
        Tensor g = t.grad();
        if (!g.defined()) fail(PyExc_RuntimeError, "ClipAdamW.step(): a parameter has no gradient");
        if (g.scalar_type() != at::kFloat || !g.is_contiguous()) {
            g = g.to(at::kFloat).contiguous();
            t.mutable_grad() = g;
        }
        p[i] = reinterpret_cast<uint64_t>(g.const_data_ptr());
    }
    bytes_guard.o = nullptr;
    return bytes;
}
// bump_versions(params): what an in-place operation would have done to the version counters
PyObject* bump_versions(PyObject* const* a) {
    PyObject* seq = PySequence_Fast(a[0], "a sequence of parameters is expected");
    if (!seq) throw PyError{};
    struct Guard { PyObject* o; ~Guard() { Py_DECREF(o); } } guard{seq};
    for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(seq); ++i) tensor_arg(PySequence_Fast_GET_ITEM(seq, i)).unsafeGetTensorImpl()->bump_version();
    Py_RETURN_NONE;
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
    JF_ENTRY(layernorm_forward, 5), JF_ENTRY(layernorm_backward, 11), JF_ENTRY(add, 9), JF_ENTRY(linear_forward, 5),
    JF_ENTRY(linear_wgrad, 6), JF_ENTRY(linear_backward, 13), JF_ENTRY(quantize_parts, 5), JF_ENTRY(attention_forward, 2),
    JF_ENTRY(attention_backward, 11), JF_ENTRY(embed_forward, 3), JF_ENTRY(embed_backward, 5), JF_ENTRY(final_norm_forward, 3),
    JF_ENTRY(final_norm_backward, 6), JF_ENTRY(lm_loss_forward, 2), JF_ENTRY(lm_loss_backward, 5), JF_ENTRY(gradient_pointers, 1),
    JF_ENTRY(bump_versions, 1), {"set_error_class", set_error_class, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host_ops", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host_ops(void) { return PyModule_Create(&module); }
