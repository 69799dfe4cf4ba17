// CPython entry points for the calls that a host program issues one at a time on torch tensors: argument checks, output
// and workspace allocation, the current stream and the library call, in one native function each.
//
// The same steps in Python (attribute checks, torch.empty, the current stream, a ctypes call with eight arguments) take 8 to
// 25 us per call, more than the kernels of a small projection: one 8192 x 2048 W4A16 GEMV is 4.4 us on the device.
//
// Every function takes positional arguments only (METH_FASTCALL) and keeps the checks and error types of the Python
// wrappers: ValueError for a tensor that is not on a CUDA device or not contiguous, TypeError for its type, and the status
// of the library through the callable registered with set_raise().
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../../include/nve_kernels.h"

namespace {

PyObject* g_raise = nullptr;                    // raise_status(name, status): raises the Python error of a library status
PyObject* g_oom = nullptr;                      // torch.OutOfMemoryError
thread_local unsigned long long t_capture = 0;  // stream that records the library's graph on this thread, 0 = none

nve_stream_t current_stream() {
    if (t_capture != 0) return reinterpret_cast<nve_stream_t>(t_capture);
    return c10::cuda::getCurrentCUDAStream().stream();
}

// A step of a call failed and the Python error is set.
struct Failed {};

[[noreturn]] void fail(PyObject* type, const char* fmt, const char* name) {
    PyErr_Format(type, fmt, name);
    throw Failed();
}

const at::Tensor& tensor(PyObject* o, const char* name) {
    if (!THPVariable_Check(o)) fail(PyExc_TypeError, "%s must be a tensor", name);
    return THPVariable_Unpack(o);
}
void* cuda_ptr(const at::Tensor& t, const char* name) {
    if (!t.is_cuda()) fail(PyExc_ValueError, "%s must be a CUDA tensor", name);
    if (!t.is_contiguous()) fail(PyExc_ValueError, "%s must be contiguous", name);
    return t.data_ptr();
}
void* typed_ptr(const at::Tensor& t, at::ScalarType type, const char* name) {
    void* p = cuda_ptr(t, name);
    if (t.scalar_type() != type) fail(PyExc_TypeError, "%s has the wrong dtype", name);
    return p;
}
void* codes_ptr(const at::Tensor& t, const char* name) {
    void* p = cuda_ptr(t, name);
    if (t.scalar_type() != at::kChar && t.scalar_type() != at::kByte) fail(PyExc_TypeError, "%s has the wrong dtype", name);
    return p;
}
void* optional_ptr(PyObject* o, at::ScalarType type, const char* name) {
    return o == Py_None ? nullptr : typed_ptr(tensor(o, name), type, name);
}
int act_dtype(const at::Tensor& t, const char* name) {
    if (t.scalar_type() == at::kHalf) return NVE_DT_F16;
    if (t.scalar_type() == at::kBFloat16) return NVE_DT_BF16;
    fail(PyExc_TypeError, "%s has the wrong dtype", name);
}
long integer(PyObject* o) {
    const long v = PyLong_AsLong(o);
    if (v == -1 && PyErr_Occurred()) throw Failed();
    return v;
}
double number(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw Failed();
    return v;
}
void expect(Py_ssize_t have, Py_ssize_t want, const char* name) {
    if (have != want) fail(PyExc_TypeError, "%s: wrong number of arguments", name);
}
void status(const char* name, int st) {
    if (st == NVE_OK) return;
    if (g_raise != nullptr) {
        PyObject* r = PyObject_CallFunction(g_raise, "si", name, st);
        Py_XDECREF(r);
    }
    if (!PyErr_Occurred()) PyErr_Format(PyExc_RuntimeError, "%s: status %d", name, st);
    throw Failed();
}
// Other Python threads run while this one allocates and launches: either can wait for the device (a full launch queue, an allocation
// that has to free memory first).
struct WithoutGil {
    PyThreadState* state = PyEval_SaveThread();
    ~WithoutGil() { PyEval_RestoreThread(state); }
};
at::Tensor empty(at::IntArrayRef size, at::ScalarType type, const at::Tensor& like) {
    return at::detail::empty_cuda(size, type, like.device(), c10::nullopt);
}
PyObject* wrap(at::Tensor t) { return THPVariable_Wrap(std::move(t)); }

template <class F> PyObject* guarded(F f) {
    try {
        return f();
    } catch (const Failed&) {
        return nullptr;
    } catch (const c10::OutOfMemoryError& e) {
        PyErr_SetString(g_oom != nullptr ? g_oom : PyExc_MemoryError, e.what_without_backtrace());
        return nullptr;
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

// matvec_w4a16(x, nibbles, scales, awq | None, n, k) -> [1, n] f16
PyObject* matvec_w4a16(PyObject*, PyObject* const* a, Py_ssize_t na) {
    return guarded([&] {
        expect(na, 6, "matvec_w4a16");
        const at::Tensor& x = tensor(a[0], "x");
        const auto* xp = static_cast<const uint16_t*>(typed_ptr(x, at::kHalf, "x"));
        const auto* nib = static_cast<const uint8_t*>(typed_ptr(tensor(a[1], "nibbles"), at::kByte, "nibbles"));
        const auto* sc = static_cast<const float*>(typed_ptr(tensor(a[2], "scales"), at::kFloat, "scales"));
        const auto* awq = static_cast<const float*>(optional_ptr(a[3], at::kFloat, "awq"));
        const long n = integer(a[4]), k = integer(a[5]);
        at::Tensor out;
        int st;
        {
            WithoutGil others;
            out = empty({1, n}, at::kHalf, x);
            nve_matvec_w4a16(xp, nib, sc, awq, static_cast<uint16_t*>(out.data_ptr()), static_cast<int>(n), static_cast<int>(k), current_stream());
            st = nve_b200_last_status();
        }
        status("nve_matvec_w4a16", st);
        return wrap(std::move(out));
    });
}

// quantize_f16_q8(x) -> (codes [K] int8, scales [K/32] f32)
PyObject* quantize_f16_q8(PyObject*, PyObject* const* a, Py_ssize_t na) {
    return guarded([&] {
        expect(na, 1, "quantize_f16_q8");
        const at::Tensor& x = tensor(a[0], "x");
        const int64_t k = x.numel();
        if (k % 32 != 0) fail(PyExc_ValueError, "%s: K must be multiple of 32", "quantize_f16_q8");
        const auto* xp = static_cast<const uint16_t*>(typed_ptr(x, at::kHalf, "x"));
        at::Tensor xq, xs;
        int st;
        {
            WithoutGil others;
            xq = empty({k}, at::kChar, x);
            xs = empty({k / 32}, at::kFloat, x);
            nve_quantize_f16_q8(xp, static_cast<int8_t*>(xq.data_ptr()), static_cast<float*>(xs.data_ptr()), static_cast<int>(k), current_stream());
            st = nve_b200_last_status();
        }
        status("nve_quantize_f16_q8", st);
        PyObject* r = PyTuple_New(2);
        PyTuple_SET_ITEM(r, 0, wrap(std::move(xq)));
        PyTuple_SET_ITEM(r, 1, wrap(std::move(xs)));
        return r;
    });
}

// matvec_w4a8(codes, code scales, nibbles, scales, n, k) -> [1, n] f16
PyObject* matvec_w4a8(PyObject*, PyObject* const* a, Py_ssize_t na) {
    return guarded([&] {
        expect(na, 6, "matvec_w4a8");
        const at::Tensor& xq = tensor(a[0], "xq");
        const auto* qp = static_cast<const int8_t*>(codes_ptr(xq, "xq"));
        const auto* qs = static_cast<const float*>(typed_ptr(tensor(a[1], "xq_scales"), at::kFloat, "xq_scales"));
        const auto* nib = static_cast<const uint8_t*>(typed_ptr(tensor(a[2], "nibbles"), at::kByte, "nibbles"));
        const auto* sc = static_cast<const float*>(typed_ptr(tensor(a[3], "wt_scales"), at::kFloat, "wt_scales"));
        const long n = integer(a[4]), k = integer(a[5]);
        at::Tensor out;
        int st;
        {
            WithoutGil others;
            out = empty({1, n}, at::kHalf, xq);
            nve_matvec_w4a8(qp, qs, nib, sc, static_cast<uint16_t*>(out.data_ptr()), static_cast<int>(n), static_cast<int>(k), current_stream());
            st = nve_b200_last_status();
        }
        status("nve_matvec_w4a8", st);
        return wrap(std::move(out));
    });
}

// gemm_w4a16_wide(x, ((nibbles, scales, n), ...), k, outs | None, scratch | None) -> list of outputs [M, n] of x's type
PyObject* gemm_w4a16_wide(PyObject*, PyObject* const* a, Py_ssize_t na) {
    return guarded([&]() -> PyObject* {
        expect(na, 5, "gemm_w4a16_wide");
        const at::Tensor& x = tensor(a[0], "x");
        const void* xp = cuda_ptr(x, "x");
        const int dt = act_dtype(x, "x");
        if (x.dim() != 2) fail(PyExc_ValueError, "%s must be [M, K]", "x");
        const int64_t m = x.size(0);
        const int k = static_cast<int>(integer(a[2]));
        if (x.size(1) != k) fail(PyExc_ValueError, "%s: x must be [M, k]", "gemm_w4a16_wide");
        struct Ref {
            PyObject* o = nullptr;
            ~Ref() { Py_XDECREF(o); }
        } ws, outs;
        ws.o = PySequence_Fast(a[1], "weights");
        if (ws.o == nullptr) throw Failed();
        const Py_ssize_t count = PySequence_Fast_GET_SIZE(ws.o);
        if (a[3] != Py_None && (outs.o = PySequence_Fast(a[3], "outs")) == nullptr) throw Failed();
        if (count < 1 || count > 3 || (outs.o != nullptr && PySequence_Fast_GET_SIZE(outs.o) != count))
            fail(PyExc_ValueError, "%s: one to three matrices, one output each", "gemm_w4a16_wide");
        nve_b200_w4_matrix mats[3];
        at::Tensor made[3];
        int ns[3];
        for (Py_ssize_t i = 0; i < count; i++) {
            PyObject* w = PySequence_Fast_GET_ITEM(ws.o, i);
            if (!PyTuple_Check(w) || PyTuple_GET_SIZE(w) != 3) fail(PyExc_TypeError, "%s: a matrix is (nibbles, scales, n)", "gemm_w4a16_wide");
            mats[i].nibbles = static_cast<const uint8_t*>(typed_ptr(tensor(PyTuple_GET_ITEM(w, 0), "nibbles"), at::kByte, "nibbles"));
            mats[i].scales = static_cast<const float*>(typed_ptr(tensor(PyTuple_GET_ITEM(w, 1), "scales"), at::kFloat, "scales"));
            mats[i].residual = nullptr;
            mats[i].N = ns[i] = static_cast<int>(integer(PyTuple_GET_ITEM(w, 2)));
            if (outs.o != nullptr) {
                made[i] = tensor(PySequence_Fast_GET_ITEM(outs.o, i), "out");
                typed_ptr(made[i], x.scalar_type(), "out");
            }
        }
        void* scratch = nullptr;
        size_t bytes = 0;
        if (a[4] != Py_None) {
            const at::Tensor& s = tensor(a[4], "scratch");
            scratch = cuda_ptr(s, "scratch");
            bytes = s.nbytes();
        }
        int st;
        at::Tensor own;
        {
            WithoutGil others;
            for (Py_ssize_t i = 0; i < count; i++) {
                if (outs.o == nullptr) made[i] = empty({m, ns[i]}, x.scalar_type(), x);
                mats[i].out = made[i].data_ptr();
            }
            if (a[4] == Py_None) {
                bytes = nve_b200_gemm_w4a16_multi_scratch_bytes(static_cast<int>(m), ns, static_cast<int>(count), k);
                if (bytes > 0) {
                    own = empty({static_cast<int64_t>(bytes)}, at::kByte, x);
                    scratch = own.data_ptr();
                }
            }
            st = nve_b200_gemm_w4a16_wide(xp, dt, mats, static_cast<int>(count), dt, static_cast<int>(m), k, scratch, bytes, current_stream());
        }
        status("nve_b200_gemm_w4a16_wide", st);
        PyObject* r = PyList_New(count);
        for (Py_ssize_t i = 0; i < count; i++) PyList_SET_ITEM(r, i, wrap(std::move(made[i])));
        return r;
    });
}

// q4_quantize(w [n, k] f32, awq | None) -> (nibbles [n, k/2] uint8, scales [n, k/32] f32)
PyObject* q4_quantize(PyObject*, PyObject* const* a, Py_ssize_t na) {
    return guarded([&] {
        expect(na, 2, "q4_quantize");
        const at::Tensor& w = tensor(a[0], "W");
        if (w.dim() != 2) fail(PyExc_ValueError, "%s must be [n, k]", "W");
        const int64_t n = w.size(0), k = w.size(1);
        const auto* wp = static_cast<const float*>(typed_ptr(w, at::kFloat, "W"));
        const auto* awq = static_cast<const float*>(optional_ptr(a[1], at::kFloat, "awq_scales"));
        at::Tensor nib, sc;
        int st;
        {
            WithoutGil others;
            nib = empty({n, k / 2}, at::kByte, w);
            sc = empty({n, k / 32}, at::kFloat, w);
            st = nve_b200_q4_quantize(wp, awq, static_cast<uint8_t*>(nib.data_ptr()), static_cast<float*>(sc.data_ptr()), static_cast<int>(n),
                                      static_cast<int>(k), current_stream());
        }
        status("nve_b200_q4_quantize", st);
        PyObject* r = PyTuple_New(2);
        PyTuple_SET_ITEM(r, 0, wrap(std::move(nib)));
        PyTuple_SET_ITEM(r, 1, wrap(std::move(sc)));
        return r;
    });
}

// prefill_layer(hidden [S, H] f16, ((nibbles, scales, n, k) of q, k, v, o, gate, up, down), input norm, post-attention norm, K cache, V cache,
//               rope cos, rope sin, heads, KV heads, head_dim, max_seq, eps, scale, start_pos) -> [S, H] f16, or None where the
// sizes do not fit together or the library does not cover them: the caller then issues the launches one by one.
PyObject* prefill_layer(PyObject*, PyObject* const* a, Py_ssize_t na) {
    return guarded([&]() -> PyObject* {
        expect(na, 15, "prefill_layer");
        const at::Tensor& x = tensor(a[0], "hidden");
        const auto* xp = static_cast<const uint16_t*>(typed_ptr(x, at::kHalf, "hidden"));
        if (x.dim() != 2) fail(PyExc_ValueError, "%s must be [S, hidden]", "hidden");
        if (!PyTuple_Check(a[1]) || PyTuple_GET_SIZE(a[1]) != 7) fail(PyExc_TypeError, "%s: seven projections", "prefill_layer");
        const int64_t rows = x.size(0), h = x.size(1), nh = integer(a[8]), nkv = integer(a[9]), hd = integer(a[10]), max_seq = integer(a[11]);
        nve_b200_rows_layer L;
        int64_t n[7], k[7];
        bool fits = rows <= 65535 && h <= 0x7FFFFFFF && nh > 0 && nkv > 0 && nh <= 65536 && nkv <= 65536 && hd > 0 && hd <= 65536 && max_seq > 0 &&
                    max_seq <= 0x7FFFFFFF;
        for (int i = 0; i < 7; i++) {
            PyObject* p = PyTuple_GET_ITEM(a[1], i);
            if (!PyTuple_Check(p) || PyTuple_GET_SIZE(p) != 4) fail(PyExc_TypeError, "%s: a projection is (nibbles, scales, n, k)", "prefill_layer");
            const at::Tensor &nib = tensor(PyTuple_GET_ITEM(p, 0), "nibbles"), &sc = tensor(PyTuple_GET_ITEM(p, 1), "scales");
            L.nibbles[i] = static_cast<const uint8_t*>(typed_ptr(nib, at::kByte, "nibbles"));
            L.scales[i] = static_cast<const float*>(typed_ptr(sc, at::kFloat, "scales"));
            n[i] = integer(PyTuple_GET_ITEM(p, 2));
            k[i] = integer(PyTuple_GET_ITEM(p, 3));
            fits = fits && n[i] > 0 && n[i] <= 0x7FFFFFFF && k[i] > 0 && k[i] <= 0x7FFFFFFF && nib.numel() == n[i] * k[i] / 2 && sc.numel() == n[i] * k[i] / 32;
        }
        const int64_t q = nh * hd, kv = nkv * hd, ffn = n[4];
        const int64_t want_n[7] = {q, kv, kv, h, ffn, ffn, h}, want_k[7] = {h, h, h, q, h, h, ffn};
        for (int i = 0; i < 7; i++) fits = fits && n[i] == want_n[i] && k[i] == want_k[i];
        auto vec = [&](int i, const char* name, int64_t least, bool exact) {
            const at::Tensor& t = tensor(a[i], name);
            fits = fits && (exact ? t.numel() == least : t.numel() >= least);
            return static_cast<uint16_t*>(typed_ptr(t, at::kHalf, name));
        };
        L.input_norm = vec(2, "input norm", h, true);
        L.post_attn_norm = vec(3, "post-attention norm", h, true);
        L.k_cache = vec(4, "k cache", kv * max_seq, true);
        L.v_cache = vec(5, "v cache", kv * max_seq, true);
        L.rope_cos = vec(6, "rope cos", max_seq * (hd / 2), false);
        L.rope_sin = vec(7, "rope sin", max_seq * (hd / 2), false);
        L.norm_eps = static_cast<float>(number(a[12]));
        L.attn_scale = static_cast<float>(number(a[13]));
        const int64_t start = integer(a[14]);
        at::Tensor out;
        int st = NVE_OK;
        if (fits && start >= 0 && start + rows <= max_seq) {
            L.hidden = static_cast<int>(h);
            L.ffn = static_cast<int>(ffn);
            L.num_heads = static_cast<int>(nh);
            L.num_kv_heads = static_cast<int>(nkv);
            L.head_dim = static_cast<int>(hd);
            L.max_seq = static_cast<int>(max_seq);
            WithoutGil others;
            if (const size_t need = nve_b200_prefill_layer_workspace_bytes(&L, static_cast<int>(rows)); need > 0) {
                at::Tensor ws = empty({static_cast<int64_t>(need)}, at::kByte, x);  // blocks of the caching allocator are 512-byte aligned
                out = empty({rows, h}, at::kHalf, x);
                st = nve_b200_prefill_layer(&L, xp, static_cast<uint16_t*>(out.data_ptr()), static_cast<int>(rows), static_cast<int>(start), ws.data_ptr(),
                                            need, current_stream());
            }
        }
        status("nve_b200_prefill_layer", st);
        if (!out.defined()) Py_RETURN_NONE;
        return wrap(std::move(out));
    });
}

// set_capture_stream(stream | 0): where this thread's calls go while a graph is recorded
PyObject* set_capture_stream(PyObject*, PyObject* const* a, Py_ssize_t na) {
    return guarded([&] {
        expect(na, 1, "set_capture_stream");
        const unsigned long long s = PyLong_AsUnsignedLongLong(a[0]);
        if (PyErr_Occurred()) throw Failed();
        t_capture = s;
        Py_INCREF(Py_None);
        return Py_None;
    });
}

// set_raise(callable, torch.OutOfMemoryError)
PyObject* set_raise(PyObject*, PyObject* const* a, Py_ssize_t na) {
    return guarded([&] {
        expect(na, 2, "set_raise");
        Py_INCREF(a[0]);
        Py_XDECREF(g_raise);
        g_raise = a[0];
        Py_INCREF(a[1]);
        Py_XDECREF(g_oom);
        g_oom = a[1];
        Py_INCREF(Py_None);
        return Py_None;
    });
}

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {FAST(matvec_w4a16), FAST(quantize_f16_q8),    FAST(matvec_w4a8), FAST(gemm_w4a16_wide),
                          FAST(q4_quantize),  FAST(prefill_layer),      FAST(set_capture_stream), FAST(set_raise), {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host", "torch-tensor calls into libnve_kernels.so", -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&kModule); }
