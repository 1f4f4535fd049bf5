// sl8_torch.cpp -- the device-operand calls of layers.py from torch tensors to the C ABI without Python in between.
//
// A layer of a small problem takes less time on the GPU than reading a dozen tensor attributes through Python and
// converting seventeen arguments through ctypes (about 9 us a call).  Each function here checks what the method of
// the same name checks, and launches.  It returns the output, or the negative status of the C ABI as an int, or None:
// whatever it does not take as it stands (another type of tensor, an operand out of place, an error to be raised) is
// left to the method, which does the same through Python and raises.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <climits>

#include "../../include/siglip_fp8.h"

namespace {

// Arguments of one call, taken from the front.  `ok` falls to false at the first one that is not the plain case.
struct Args {
    PyObject* const* v;
    Py_ssize_t n, at = 0;
    sl8_handle_t h = nullptr;
    int device = 0;
    bool ok = true;

    Args(PyObject* const* args, Py_ssize_t count, Py_ssize_t want) : v(args), n(count) {
        ok = count == want + 3;
        if (!ok) return;
        h = static_cast<sl8_handle_t>(reinterpret_cast<void*>(PyLong_AsSize_t(v[at++])));
        device = static_cast<int>(PyLong_AsLong(v[at++]));
        current = v[at] == Py_None;
        if (!current) given_stream = reinterpret_cast<void*>(PyLong_AsSize_t(v[at]));
        at++;
        if (PyErr_Occurred()) PyErr_Clear(), ok = false;
        if (!h) ok = false;
    }
    // The stream given, or torch's current one (asked for only when the operands are known to be on the GPU).
    sl8_stream_t stream() const {
        return current ? static_cast<sl8_stream_t>(c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream()) : given_stream;
    }
    // A temporary of this call that its stream still uses when the call returns and the temporary goes.
    void outlives(const at::Tensor& t) const {
        if (!current) t.record_stream(c10::cuda::getStreamFromExternal(static_cast<cudaStream_t>(given_stream), static_cast<c10::DeviceIndex>(device)));
    }
    // A plain strided tensor on the handle's GPU (subclasses, wrappers of a transform and the like go through Python).
    const at::Tensor* tensor() { return plain(v[at++]); }
    const at::Tensor* optional(bool& given) {
        PyObject* o = v[at++];
        given = o != Py_None;
        return given ? plain(o) : nullptr;
    }
    // `n` fp32 values in a row, or None.
    const float* floats(int64_t n) {
        bool given;
        const at::Tensor* t = optional(given);
        if (!t) return nullptr;
        if (t->scalar_type() != at::kFloat || t->numel() < n || (n > 1 && !t->is_contiguous())) { ok = false; return nullptr; }
        return static_cast<const float*>(t->const_data_ptr());
    }
    const float* scale() { return floats(1); }
    long long integer() {
        PyObject* o = v[at++];
        if (!PyLong_CheckExact(o)) { ok = false; return 0; }
        int overflow = 0;
        const long long x = PyLong_AsLongLongAndOverflow(o, &overflow);
        if (overflow || x > INT_MAX || x < INT_MIN) ok = false;
        return x;
    }
    double real() {
        PyObject* o = v[at++];
        if (!PyFloat_CheckExact(o)) { ok = false; return 0; }
        return PyFloat_AS_DOUBLE(o);
    }

  private:
    bool current = true;
    sl8_stream_t given_stream = nullptr;

    const at::Tensor* plain(PyObject* o) {
        if (!THPVariable_CheckExact(o)) { ok = false; return nullptr; }
        const at::Tensor& t = THPVariable_Unpack(o);
        if (!t.defined() || !t.has_storage() || t.layout() != at::kStrided || !t.is_cuda() || t.device().index() != device ||
            t.key_set().has(c10::DispatchKey::Python) || t.key_set().has(c10::DispatchKey::Functionalize)) {
            ok = false;
            return nullptr;
        }
        return &t;
    }
};

inline bool codes(const at::Tensor& t) { return t.scalar_type() == at::kByte || t.scalar_type() == at::kFloat8_e4m3fn; }
inline bool matrix(const at::Tensor& t) { return t.dim() == 2 && t.stride(1) == 1; }
inline bool shaped(const at::Tensor& t, int64_t rows, int64_t cols) { return matrix(t) && t.size(0) == rows && t.size(1) == cols; }

// A [M, K] and B [N, K], e4m3, K contiguous.
struct Gemm {
    const at::Tensor *A, *B;
    int64_t M = 0, N = 0, K = 0;
    Gemm(Args& a) {
        A = a.tensor();
        B = a.ok ? a.tensor() : nullptr;
        if (!a.ok) return;
        a.ok = codes(*A) && codes(*B) && matrix(*A) && matrix(*B) && A->size(1) == B->size(1) && B->size(0) <= INT_MAX && A->size(1) <= INT_MAX;
        if (a.ok) { M = A->size(0); N = B->size(0); K = A->size(1); }
    }
};

// A bias of n elements (bf16, or fp32 with the flag), or none: what the kernel reads.  The flag and the type must not contradict.
const void* bias_of(Args& a, const at::Tensor* t, int64_t n, unsigned& flags) {
    if (!a.ok || !t) return nullptr;
    const bool f32 = t->scalar_type() == at::kFloat;
    if (f32) flags |= SL8_FLAG_BIAS_F32;
    if ((!f32 && (t->scalar_type() != at::kBFloat16 || (flags & SL8_FLAG_BIAS_F32))) || t->numel() < n || !t->is_contiguous()) a.ok = false;
    return a.ok ? t->const_data_ptr() : nullptr;
}

// `out`, or a new [M, N] beside A.  Defined unless the call is not the plain case.
at::Tensor output(Args& a, const at::Tensor* given, const at::Tensor& A, int64_t M, int64_t N, at::ScalarType type, bool e4m3_too) {
    if (!given) return at::empty({M, N}, A.options().dtype(type));
    const bool typed = given->scalar_type() == at::kBFloat16 || (e4m3_too && codes(*given));
    if (!typed || !shaped(*given, M, N)) a.ok = false;
    return *given;
}

// Whether t has room for [rows, cols] codes at its own row pitch.
bool holds_codes(const at::Tensor& t, int64_t rows, int64_t cols) {
    return codes(t) && t.dim() == 2 && t.size(0) >= rows && t.size(1) >= cols && (t.stride(1) == 1 || t.size(1) == 1);
}

// `out`, or new codes beside x: [rows, cols] of rows on 128-byte lines.  Undefined if `out` has no room for them.
at::Tensor codes_into(const at::Tensor* given, const at::Tensor& x, int64_t rows, int64_t cols) {
    if (!given) return at::empty({rows, (cols + 127) / 128 * 128}, x.options().dtype(at::kByte)).narrow(1, 0, cols);
    return holds_codes(*given, rows, cols) ? *given : at::Tensor();
}

PyObject* result(int rc, const at::Tensor& out) {
    if (rc != SL8_OK) return PyLong_FromLong(rc);
    return THPVariable_Wrap(out);
}

// The status of `entry`, a function of the C ABI, with the interpreter lock released.  The arguments are numbers and addresses,
// read from the tensors while the lock is held: that may throw (a tensor without memory, no driver), and an exception must not
// leave the part without the lock; nor may another thread change a tensor halfway through its reading.
template <typename... P, typename... V>
int unlocked(int (*entry)(P...), V... values) {
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = entry(values...);
    Py_END_ALLOW_THREADS
    return rc;
}

#define SL8_PY(name) PyObject* name(PyObject*, PyObject* const* args, Py_ssize_t count)

// h, device, stream, A, B, bias, scale_a, scale_b, out_scale, out, type of a new out (0 bf16, 1 float8_e4m3fn, 2 uint8), flags
SL8_PY(linear) {
    HANDLE_TH_ERRORS
    Args a(args, count, 9);
    if (!a.ok) Py_RETURN_NONE;
    Gemm g(a);
    if (!a.ok) Py_RETURN_NONE;
    bool has_bias, has_out;
    const at::Tensor* bias = a.optional(has_bias);
    const float *sa = a.scale(), *sb = a.scale(), *so = a.scale();
    const at::Tensor* given = a.optional(has_out);
    const long long new_type = a.integer();
    unsigned flags = static_cast<unsigned>(a.integer());
    const void* const b = bias_of(a, bias, g.N, flags);
    if (!a.ok) Py_RETURN_NONE;
    const at::Tensor out = output(a, given, *g.A, g.M, g.N, new_type == 0 ? at::kBFloat16 : new_type == 1 ? at::kFloat8_e4m3fn : at::kByte, true);
    if (!a.ok) Py_RETURN_NONE;
    const int type = codes(out) ? SL8_OUT_E4M3 : SL8_OUT_BF16;
    const int rc = unlocked(sl8_fc1_gelu_fp8, a.h, g.A->const_data_ptr(), g.A->stride(0), g.B->const_data_ptr(), g.B->stride(0), sa, sb,
                            b, out.mutable_data_ptr(), out.stride(0), type, so, g.M,
                            static_cast<int>(g.N), static_cast<int>(g.K), flags, a.stream());
    return result(rc, out);
    END_HANDLE_TH_ERRORS
}

// h, device, stream, A, B, table, scale_a, scale_b, out, period (None: the table's rows), row_phase, flags
SL8_PY(patch_embed) {
    HANDLE_TH_ERRORS
    Args a(args, count, 9);
    if (!a.ok) Py_RETURN_NONE;
    Gemm g(a);
    if (!a.ok) Py_RETURN_NONE;
    const at::Tensor* table = a.tensor();
    const float *sa = a.scale(), *sb = a.scale();
    bool has_out;
    const at::Tensor* given = a.optional(has_out);
    const bool whole = a.v[a.at] == Py_None;
    long long period = 0;
    if (whole) a.at++;
    else period = a.integer();
    const long long row_phase = a.integer();
    const unsigned flags = static_cast<unsigned>(a.integer());
    if (!a.ok || table->scalar_type() != at::kBFloat16 || !matrix(*table) || table->size(1) != g.N || table->size(0) > INT_MAX) Py_RETURN_NONE;
    if (whole) period = table->size(0);
    const at::Tensor out = output(a, given, *g.A, g.M, g.N, at::kBFloat16, false);
    if (!a.ok) Py_RETURN_NONE;
    const int rc = unlocked(sl8_patch_embed_fp8, a.h, g.A->const_data_ptr(), g.A->stride(0), g.B->const_data_ptr(), g.B->stride(0), sa, sb, table->const_data_ptr(),
                            table->stride(0), static_cast<int>(period), static_cast<int>(table->size(0)), static_cast<int>(row_phase),
                            out.mutable_data_ptr(), out.stride(0), g.M, static_cast<int>(g.N), static_cast<int>(g.K), flags, a.stream());
    return result(rc, out);
    END_HANDLE_TH_ERRORS
}

// h, device, stream, A, B, bias, residual, scale_a, scale_b, out, flags
SL8_PY(fc2_residual) {
    HANDLE_TH_ERRORS
    Args a(args, count, 8);
    if (!a.ok) Py_RETURN_NONE;
    Gemm g(a);
    if (!a.ok) Py_RETURN_NONE;
    bool has_bias, has_out;
    const at::Tensor* bias = a.optional(has_bias);
    const at::Tensor* residual = a.tensor();
    const float *sa = a.scale(), *sb = a.scale();
    const at::Tensor* given = a.optional(has_out);
    unsigned flags = static_cast<unsigned>(a.integer());
    const void* const b = bias_of(a, bias, g.N, flags);
    if (!a.ok || residual->scalar_type() != at::kBFloat16 || !shaped(*residual, g.M, g.N)) Py_RETURN_NONE;
    const at::Tensor out = output(a, given, *g.A, g.M, g.N, at::kBFloat16, false);
    if (!a.ok) Py_RETURN_NONE;
    const int rc = unlocked(sl8_fc2_residual_fp8, a.h, g.A->const_data_ptr(), g.A->stride(0), g.B->const_data_ptr(), g.B->stride(0), sa, sb,
                            b, residual->const_data_ptr(), residual->stride(0), out.mutable_data_ptr(),
                            out.stride(0), g.M, static_cast<int>(g.N), static_cast<int>(g.K), flags, a.stream());
    return result(rc, out);
    END_HANDLE_TH_ERRORS
}

// h, device, stream, A, W1, bias1, W2, bias2, residual, scale_a, scale_w1, scale_w2, hidden_scale, hidden, out, flags
SL8_PY(mlp_chain) {
    HANDLE_TH_ERRORS
    Args a(args, count, 13);
    if (!a.ok) Py_RETURN_NONE;
    Gemm g(a);                                   // [M, d_model] x [d_ff, d_model]
    if (!a.ok) Py_RETURN_NONE;
    bool has_b1, has_b2, has_hidden, has_out;
    const at::Tensor* bias1 = a.optional(has_b1);
    const at::Tensor* W2 = a.tensor();
    const at::Tensor* bias2 = a.optional(has_b2);
    const at::Tensor* residual = a.tensor();
    const float *sa = a.scale(), *s1 = a.scale(), *s2 = a.scale();
    const float* sh = a.scale();
    const at::Tensor* hidden = a.optional(has_hidden);
    const at::Tensor* given = a.optional(has_out);
    unsigned flags = static_cast<unsigned>(a.integer());
    if (!a.ok || !sh || !codes(*W2) || !shaped(*W2, g.K, g.N) || residual->scalar_type() != at::kBFloat16 || !shaped(*residual, g.M, g.K) ||
        (has_hidden && (!codes(*hidden) || !shaped(*hidden, g.M, g.N))))
        Py_RETURN_NONE;
    // One flag speaks for both: it is known before either is looked at.
    if ((has_b1 && bias1->scalar_type() == at::kFloat) || (has_b2 && bias2->scalar_type() == at::kFloat)) flags |= SL8_FLAG_BIAS_F32;
    const void *const b1 = bias_of(a, bias1, g.N, flags), *const b2 = bias_of(a, bias2, g.K, flags);
    const at::Tensor out = output(a, given, *g.A, g.M, g.K, at::kBFloat16, false);
    if (!a.ok) Py_RETURN_NONE;
    const at::Tensor scratch = codes_into(hidden, *g.A, g.M, g.N);
    if (!hidden) a.outlives(scratch);
    const int rc = unlocked(sl8_mlp_chain_fp8, a.h, g.A->const_data_ptr(), g.A->stride(0), g.B->const_data_ptr(), g.B->stride(0), sa, s1,
                            b1, scratch.mutable_data_ptr(), scratch.stride(0),
                            sh, W2->const_data_ptr(), W2->stride(0), s2,
                            b2, residual->const_data_ptr(), residual->stride(0), out.mutable_data_ptr(),
                            out.stride(0), g.M, static_cast<int>(g.K), static_cast<int>(g.N), flags, a.stream());
    return result(rc, out);
    END_HANDLE_TH_ERRORS
}

// SL8_DT_* of an activation, or -1.
int activation(const at::Tensor& t) { return t.scalar_type() == at::kFloat ? SL8_DT_F32 : t.scalar_type() == at::kBFloat16 ? SL8_DT_BF16 : -1; }
// Rows of an activation, one element after the other, at a pitch of stride(0).
bool rows_of(const at::Tensor& t) { return t.dim() == 2 && (t.stride(1) == 1 || t.size(1) == 1) && t.size(1) <= INT_MAX && activation(t) >= 0; }

// h, device, stream, pixels, scale, out, patch
SL8_PY(patchify_quantize) {
    HANDLE_TH_ERRORS
    Args a(args, count, 4);
    if (!a.ok) Py_RETURN_NONE;
    const at::Tensor* px = a.tensor();
    const float* scale = a.scale();
    bool has_out;
    const at::Tensor* given = a.ok ? a.optional(has_out) : nullptr;
    const long long patch = a.ok ? a.integer() : 0;
    if (!a.ok || px->dim() != 4 || !px->is_contiguous() || activation(*px) < 0 || patch < 1) Py_RETURN_NONE;
    for (int i = 0; i < 4; i++)
        if (px->size(i) > INT_MAX) Py_RETURN_NONE;
    if (px->size(2) < patch || px->size(3) < patch) Py_RETURN_NONE;
    const int64_t rows = px->size(0) * (px->size(2) / patch) * (px->size(3) / patch), cols = px->size(1) * patch * patch;
    if (rows < 1 || cols < 1) Py_RETURN_NONE;
    const at::Tensor out = codes_into(given, *px, rows, cols);
    if (!out.defined()) Py_RETURN_NONE;
    // (the kernel fills a pad of less than 128 bytes with zeros, the last row's too)
    const int64_t pitch = out.stride(0), written = pitch - cols < 128 ? pitch : (cols + 15) / 16 * 16;
    if (out.storage_offset() + (rows - 1) * pitch + written > static_cast<int64_t>(out.storage().nbytes())) Py_RETURN_NONE;
    const int rc = unlocked(sl8_patchify_quantize_e4m3, a.h, px->const_data_ptr(), activation(*px), static_cast<int>(px->size(0)), static_cast<int>(px->size(1)),
                            static_cast<int>(px->size(2)), static_cast<int>(px->size(3)), static_cast<int>(patch), scale,
                            out.mutable_data_ptr(), out.stride(0), a.stream());
    return result(rc, out);
    END_HANDLE_TH_ERRORS
}

// h, device, stream, x  ->  (amax, scale)
SL8_PY(amax_scale) {
    HANDLE_TH_ERRORS
    Args a(args, count, 1);
    if (!a.ok) Py_RETURN_NONE;
    const at::Tensor* x = a.tensor();
    if (!a.ok || !rows_of(*x)) Py_RETURN_NONE;
    const auto options = x->options().dtype(at::kFloat);
    const at::Tensor amax = at::empty({1}, options), scale = at::empty({1}, options);
    const int rc = unlocked(sl8_amax_scale, a.h, x->const_data_ptr(), activation(*x), x->size(0), static_cast<int>(x->size(1)), x->stride(0),
                            static_cast<float*>(amax.mutable_data_ptr()), static_cast<float*>(scale.mutable_data_ptr()), a.stream());
    if (rc != SL8_OK) return PyLong_FromLong(rc);
    PyObject* first = THPVariable_Wrap(amax);
    PyObject* second = first ? THPVariable_Wrap(scale) : nullptr;
    PyObject* both = second ? PyTuple_Pack(2, first, second) : nullptr;
    Py_XDECREF(first);
    Py_XDECREF(second);
    return both;
    END_HANDLE_TH_ERRORS
}

// h, device, stream, x, scale, out
SL8_PY(quantize_e4m3) {
    HANDLE_TH_ERRORS
    Args a(args, count, 3);
    if (!a.ok) Py_RETURN_NONE;
    const at::Tensor* x = a.tensor();
    const float* scale = a.scale();
    bool has_out;
    const at::Tensor* given = a.ok ? a.optional(has_out) : nullptr;
    if (!a.ok || !rows_of(*x)) Py_RETURN_NONE;
    const at::Tensor out = codes_into(given, *x, x->size(0), x->size(1));
    if (!out.defined()) Py_RETURN_NONE;
    const int rc = unlocked(sl8_quantize_e4m3, a.h, x->const_data_ptr(), activation(*x), x->size(0), static_cast<int>(x->size(1)), x->stride(0), scale,
                            out.mutable_data_ptr(), out.stride(0), a.stream());
    return result(rc, out);
    END_HANDLE_TH_ERRORS
}

// h, device, stream, x, gamma, beta, scale, out, eps
SL8_PY(layernorm_quantize) {
    HANDLE_TH_ERRORS
    Args a(args, count, 6);
    if (!a.ok) Py_RETURN_NONE;
    const at::Tensor* x = a.tensor();
    const int64_t cols = a.ok && x->dim() == 2 ? x->size(1) : 0;
    const float *gamma = a.floats(cols), *beta = a.floats(cols), *scale = a.scale();
    bool has_out;
    const at::Tensor* given = a.ok ? a.optional(has_out) : nullptr;
    const double eps = a.ok ? a.real() : 0.0;
    if (!a.ok || !rows_of(*x)) Py_RETURN_NONE;
    const at::Tensor out = codes_into(given, *x, x->size(0), x->size(1));
    if (!out.defined()) Py_RETURN_NONE;
    const int rc = unlocked(sl8_layernorm_quantize_e4m3, a.h, x->const_data_ptr(), activation(*x), x->size(0), static_cast<int>(x->size(1)), x->stride(0), gamma, beta,
                            static_cast<float>(eps), scale, out.mutable_data_ptr(), out.stride(0), a.stream());
    return result(rc, out);
    END_HANDLE_TH_ERRORS
}

#define SL8_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {SL8_METHOD(linear), SL8_METHOD(patch_embed), SL8_METHOD(fc2_residual), SL8_METHOD(mlp_chain),
                         SL8_METHOD(patchify_quantize), SL8_METHOD(amax_scale), SL8_METHOD(quantize_e4m3), SL8_METHOD(layernorm_quantize),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "sl8_torch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject* PyInit_sl8_torch(void) {
    PyObject* m = PyModule_Create(&module);
    if (m && PyModule_AddStringConstant(m, "torch_version", SL8_TORCH_VERSION) != 0) Py_CLEAR(m);     // the torch whose headers this was compiled with
    return m;
}
