// The torch side of the device entry points as a CPython extension: argument checks, output and scratch
// tensors, and the call into the C ABI, without an interpreter frame or a ctypes conversion in between.
//
// Why it exists: a decode or small prefill call keeps the GPU busy for 5 to 20 us, and the same call through
// Python checks, torch.empty and ctypes took 14 to 20 us of host time, so a token loop ran at the host's pace
// (one rope + append + attention step: 27.8 us per layer against 10.7 us of GPU time).  Here the host part of
// a call is 4 to 6 us, most of it the kernel launches themselves.
//
// Every function takes the Python wrapper's arguments in order and returns its result, or None when the call
// is not one it covers: a wrong type, a shape mismatch, a layout it would have to copy, any error status.
// The wrapper then takes its own path, which makes the copy or raises the error, so all behaviour but the speed
// is defined in one place.  Nothing is kept between calls: outputs and split-KV scratch come from torch's
// caching allocator, which orders reuse by stream.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/rustorch_attn.h"

namespace {

using at::Tensor;
constexpr auto kBf16 = at::kBFloat16;
constexpr auto kF32 = at::kFloat;

// A borrowed tensor argument; nullptr for anything else (None included).
inline const Tensor* tensor_arg(PyObject* o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }

// Optional tensor argument: false when it is neither None nor a tensor.
inline bool optional_arg(PyObject* o, const Tensor*& t) {
    t = o == Py_None ? nullptr : tensor_arg(o);
    return t || o == Py_None;
}

inline bool is(const Tensor& t, at::ScalarType type, const at::Device& dev) {
    return t.is_cuda() && t.scalar_type() == type && t.device() == dev;
}
inline bool dense(const Tensor& t, at::ScalarType type, const at::Device& dev) {
    return is(t, type, dev) && t.is_contiguous();
}
inline bool vector_of(const Tensor& t, int64_t n, const at::Device& dev) {  // int32 lengths, offsets, positions
    return dense(t, at::kInt, dev) && t.numel() == n;
}

inline bool int_arg(PyObject* o, int64_t& v, int64_t none_value) {
    if (o == Py_None) {
        v = none_value;
        return true;
    }
    if (!PyLong_Check(o)) return false;
    int overflow = 0;
    v = PyLong_AsLongLongAndOverflow(o, &overflow);
    return !overflow;
}
inline bool scale_arg(PyObject* o, float& v) {
    if (o == Py_None) {
        v = -1.f;
        return true;
    }
    if (!PyFloat_Check(o) && !PyLong_Check(o)) return false;
    const double d = PyFloat_AsDouble(o);
    if (d == -1.0 && PyErr_Occurred()) {
        PyErr_Clear();
        return false;
    }
    v = (float)d;
    return true;
}

// The truth of a flag; false for a value whose truth test raises (an array of several elements): the wrapper's own test
// raises it then.
inline bool flag_arg(PyObject* o, bool& v) {
    const int truth = PyObject_IsTrue(o);
    if (truth < 0) {
        PyErr_Clear();
        return false;
    }
    v = truth != 0;
    return true;
}

inline Tensor empty(at::IntArrayRef sizes, at::ScalarType type, const at::Device& dev) {
    return at::detail::empty_cuda(sizes, type, dev, std::nullopt);
}
template <class T = void>
inline T* ptr(const Tensor* t) {
    return t ? static_cast<T*>(t->data_ptr()) : nullptr;
}
inline PyObject* pair(const Tensor& a, const Tensor* b) {
    PyObject* x = THPVariable_Wrap(a);
    PyObject* y = b ? THPVariable_Wrap(*b) : (Py_INCREF(Py_None), Py_None);
    return Py_BuildValue("(NN)", x, y);
}

// Runs `call` (a C ABI function) with the interpreter lock released.
template <class F>
inline int unlocked(F&& call) {
    int rc;
    Py_BEGIN_ALLOW_THREADS rc = call();
    Py_END_ALLOW_THREADS return rc;
}

// C++ exceptions (an allocation that failed) become "not covered": the wrapper meets them again and raises.
template <class F>
inline PyObject* guarded(F&& body) {
    try {
        return body();
    } catch (const std::exception&) {
        if (PyErr_Occurred()) PyErr_Clear();
        Py_RETURN_NONE;
    }
}

struct DecodeArgs {
    int64_t B, Hq, Hkv, D, max_seq;
    at::Device dev = at::Device(at::kCPU);
};
inline bool decode_args(const Tensor* q, const Tensor* k, const Tensor* v, DecodeArgs& a) {
    if (!q || !k || !v || !q->is_cuda() || q->dim() != 3 || k->dim() != 4) return false;
    a.dev = q->device();
    a.B = q->size(0), a.Hq = q->size(1), a.D = q->size(2), a.Hkv = k->size(1), a.max_seq = k->size(2);
    return dense(*q, kBf16, a.dev) && dense(*k, kBf16, a.dev) && dense(*v, kBf16, a.dev) && k->size(0) == a.B &&
           k->size(3) == a.D && v->sizes() == k->sizes();
}

// q, k_cache, v_cache, kv_lens, kv_len, kv_begin, kv_end, scale, out_dtype, return_lse, workspace, out, lse
PyObject* gqa_decode(PyObject*, PyObject* const* arg, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 13) Py_RETURN_NONE;
        const Tensor *q = tensor_arg(arg[0]), *k = tensor_arg(arg[1]), *v = tensor_arg(arg[2]), *lens, *ws, *out, *lse;
        DecodeArgs a;
        int64_t kv_len, kv_begin, kv_end;
        float scale;
        bool want_lse;
        if (!decode_args(q, k, v, a) || !optional_arg(arg[3], lens) || !int_arg(arg[4], kv_len, 0) ||
            !int_arg(arg[5], kv_begin, 0) || !int_arg(arg[6], kv_end, -1) || !scale_arg(arg[7], scale) ||
            !flag_arg(arg[9], want_lse) || !optional_arg(arg[10], ws) || !optional_arg(arg[11], out) ||
            !optional_arg(arg[12], lse))
            Py_RETURN_NONE;
        if (lens && !(vector_of(*lens, a.B, a.dev) && lens->dim() == 1)) Py_RETURN_NONE;
        if (ws && !dense(*ws, at::kByte, a.dev)) Py_RETURN_NONE;
        at::ScalarType out_type = kBf16;
        Tensor new_out, new_lse, new_ws;
        if (out) {
            out_type = out->scalar_type();
            if (out->sizes() != q->sizes()) Py_RETURN_NONE;
        } else if (arg[8] != Py_None) {
            if (!THPDtype_Check(arg[8])) Py_RETURN_NONE;
            out_type = reinterpret_cast<THPDtype*>(arg[8])->scalar_type;
        }
        if (out_type != kBf16 && out_type != kF32) Py_RETURN_NONE;
        if (out && !dense(*out, out_type, a.dev)) Py_RETURN_NONE;
        if (lse && !(dense(*lse, kF32, a.dev) && lse->dim() == 2 && lse->size(0) == a.B && lse->size(1) == a.Hq))
            Py_RETURN_NONE;
        if (!out) {
            new_out = empty(q->sizes(), out_type, a.dev);
            out = &new_out;
        }
        if (!lse && want_lse) {
            new_lse = empty({a.B, a.Hq}, kF32, a.dev);
            lse = &new_lse;
        }
        if (!ws) {
            const size_t need = rt_gqa_decode_workspace_bytes(a.B, a.Hq, a.Hkv, (int)a.D, a.max_seq);
            if (need) {
                new_ws = empty({(int64_t)need}, at::kByte, a.dev);
                ws = &new_ws;
            }
        }
        void* stream = c10::cuda::getCurrentCUDAStream(a.dev.index()).stream();
        const int rc = unlocked([&] {
            return rt_gqa_decode_bf16(ptr(q), ptr(k), ptr(v), out_type == kBf16 ? ptr(out) : nullptr,
                                      out_type == kF32 ? ptr<float>(out) : nullptr, ptr<float>(lse), a.B, a.Hq, a.Hkv,
                                      (int)a.D, a.max_seq, ptr<int32_t>(lens), kv_len, kv_begin, kv_end, scale, ptr(ws),
                                      ws ? (size_t)ws->numel() : 0, stream);
        });
        if (rc != RT_OK) Py_RETURN_NONE;
        return pair(*out, lse);
    });
}

// q, k_in, v_in, k_cache, v_cache, inv_freq, pos, positions, style (RT_ROPE_*); True when done
PyObject* rope_kv_append(PyObject*, PyObject* const* arg, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 9) Py_RETURN_NONE;
        const Tensor *q = tensor_arg(arg[0]), *k_in = tensor_arg(arg[1]), *v_in = tensor_arg(arg[2]),
                     *k = tensor_arg(arg[3]), *v = tensor_arg(arg[4]), *freq = tensor_arg(arg[5]), *positions;
        DecodeArgs a;
        int64_t pos, style;
        if (!decode_args(q, k, v, a) || !k_in || !v_in || !freq || !int_arg(arg[6], pos, 0) ||
            !optional_arg(arg[7], positions) || !int_arg(arg[8], style, -1))
            Py_RETURN_NONE;
        for (const Tensor* t : {k_in, v_in})
            if (!(dense(*t, kBf16, a.dev) && t->dim() == 3 && t->size(0) == a.B && t->size(1) == a.Hkv && t->size(2) == a.D))
                Py_RETURN_NONE;
        if (!(dense(*freq, kF32, a.dev) && freq->dim() == 1 && freq->size(0) == a.D / 2)) Py_RETURN_NONE;
        if (positions && !(vector_of(*positions, a.B, a.dev) && positions->dim() == 1)) Py_RETURN_NONE;
        void* stream = c10::cuda::getCurrentCUDAStream().stream();
        const int rc = unlocked([&] {
            return rt_rope_kv_append_bf16(ptr(q), ptr(k_in), ptr(v_in), ptr(k), ptr(v), ptr<float>(freq), a.B, (int)a.Hq,
                                          (int)a.Hkv, (int)a.D, a.max_seq, pos, ptr<int32_t>(positions), (int)style, stream);
        });
        if (rc != RT_OK) Py_RETURN_NONE;
        Py_RETURN_TRUE;
    });
}

struct MaskArgs {
    const Tensor *lens = nullptr, *keep = nullptr, *offsets = nullptr;
    float scale = -1.f;
    int64_t keep_stride = 0;
};
// kv_lens, key_keep, scale, q_offsets.  Bool and uint8 keep flags are both one byte per key, zero = hidden.
inline bool mask_args(PyObject* lens, PyObject* keep, PyObject* scale, PyObject* offsets, int64_t B, int64_t Nkv,
                      const at::Device& dev, MaskArgs& m) {
    if (!optional_arg(lens, m.lens) || !optional_arg(keep, m.keep) || !optional_arg(offsets, m.offsets) ||
        !scale_arg(scale, m.scale))
        return false;
    if (m.lens && !vector_of(*m.lens, B, dev)) return false;
    if (m.offsets && !vector_of(*m.offsets, B, dev)) return false;
    if (m.keep) {
        const Tensor& t = *m.keep;
        if (!((t.scalar_type() == at::kBool || t.scalar_type() == at::kByte) && t.is_cuda() && t.device() == dev &&
              t.is_contiguous() && (t.dim() == 1 || (t.dim() == 2 && t.size(0) == B)) && t.size(-1) == Nkv))
            return false;
        m.keep_stride = t.dim() == 2 ? Nkv : 0;
    }
    return true;
}

// q, k, v, causal, kv_lens, key_keep, scale, out, lse, return_lse, q_offsets
PyObject* prefill_bf16(PyObject*, PyObject* const* arg, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 11) Py_RETURN_NONE;
        const Tensor *q = tensor_arg(arg[0]), *k = tensor_arg(arg[1]), *v = tensor_arg(arg[2]), *out, *lse;
        bool causal, want_lse;
        if (!q || !k || !v || !q->is_cuda() || q->dim() != 4 || k->dim() != 4 || !flag_arg(arg[3], causal) ||
            !optional_arg(arg[7], out) || !optional_arg(arg[8], lse) || !flag_arg(arg[9], want_lse))
            Py_RETURN_NONE;
        const at::Device dev = q->device();
        const int64_t B = q->size(0), H = q->size(1), N = q->size(2), D = q->size(3), Hkv = k->size(1), Nkv = k->size(2);
        MaskArgs m;
        if (!is(*q, kBf16, dev) || !is(*k, kBf16, dev) || !is(*v, kBf16, dev) || k->size(0) != B || k->size(3) != D ||
            v->sizes() != k->sizes() || !mask_args(arg[4], arg[5], arg[6], arg[10], B, Nkv, dev, m))
            Py_RETURN_NONE;
        if (out && !(is(*out, kBf16, dev) && out->sizes() == q->sizes())) Py_RETURN_NONE;
        if (lse && !(dense(*lse, kF32, dev) && lse->dim() == 3 && lse->size(0) == B && lse->size(1) == H && lse->size(2) == N))
            Py_RETURN_NONE;
        Tensor new_out, new_lse;
        if (!out) {  // the output takes q's layout
            new_out = q->is_non_overlapping_and_dense() ? at::detail::empty_strided_cuda(q->sizes(), q->strides(), kBf16, dev)
                                                        : empty(q->sizes(), kBf16, dev);
            out = &new_out;
        }
        if (!lse && want_lse) {
            new_lse = empty({B, H, N}, kF32, dev);
            lse = &new_lse;
        }
        int64_t strides[4][3];
        bool strided = false;
        const Tensor* all[4] = {q, k, v, out};
        for (int i = 0; i < 4; ++i) {
            if (!all[i]->is_contiguous()) strided = true;
            for (int d = 0; d < 3; ++d) strides[i][d] = all[i]->stride(d);
        }
        if (strided)
            for (const Tensor* t : all)
                if (t->numel() == 0 || t->stride(3) != 1) Py_RETURN_NONE;
        const int flags = causal ? RT_MASK_CAUSAL : RT_MASK_NONE;
        void* stream = c10::cuda::getCurrentCUDAStream().stream();
        const int rc = unlocked([&] {
            if (strided)
                return rt_attn_prefill_strided_bf16(ptr(q), ptr(k), ptr(v), ptr(out), ptr<float>(lse), B, H, Hkv, N, Nkv,
                                                    (int)D, strides[0], strides[1], strides[2], strides[3], flags,
                                                    ptr<int32_t>(m.lens), ptr<int32_t>(m.offsets), ptr<uint8_t>(m.keep),
                                                    m.keep_stride, m.scale, stream);
            if (Hkv == H && Nkv == N && !m.offsets)
                return rt_attn_prefill_bf16(ptr(q), ptr(k), ptr(v), ptr(out), ptr<float>(lse), B, H, N, (int)D, flags,
                                            ptr<int32_t>(m.lens), ptr<uint8_t>(m.keep), m.keep_stride, m.scale, stream);
            return rt_attn_prefill_gqa_bf16(ptr(q), ptr(k), ptr(v), ptr(out), ptr<float>(lse), B, H, Hkv, N, Nkv, (int)D,
                                            flags, ptr<int32_t>(m.lens), ptr<int32_t>(m.offsets), ptr<uint8_t>(m.keep),
                                            m.keep_stride, m.scale, stream);
        });
        if (rc != RT_OK) Py_RETURN_NONE;
        return pair(*out, lse);
    });
}

// q [B,T,Hq*hd], k, v [B,S,Hkv*hd], n_heads, n_kv_heads, causal, kv_lens, key_keep, scale, return_lse, q_offsets
PyObject* mha_prefill_bf16(PyObject*, PyObject* const* arg, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 11) Py_RETURN_NONE;
        const Tensor *q = tensor_arg(arg[0]), *k = tensor_arg(arg[1]), *v = tensor_arg(arg[2]);
        int64_t H, Hkv;
        bool causal, want_lse;
        if (!q || !k || !v || !q->is_cuda() || q->dim() != 3 || k->dim() != 3 || !int_arg(arg[3], H, 0) ||
            !int_arg(arg[4], Hkv, H) || H <= 0 || Hkv <= 0 || !flag_arg(arg[5], causal) || !flag_arg(arg[9], want_lse))
            Py_RETURN_NONE;
        const at::Device dev = q->device();
        const int64_t B = q->size(0), T = q->size(1), E = q->size(2), S = k->size(1), D = E / H;
        MaskArgs m;
        if (!dense(*q, kBf16, dev) || !dense(*k, kBf16, dev) || !dense(*v, kBf16, dev) || D * H != E || k->size(0) != B ||
            k->size(2) != Hkv * D || v->sizes() != k->sizes() || q->numel() == 0 || k->numel() == 0 ||
            !mask_args(arg[6], arg[7], arg[8], arg[10], B, S, dev, m))
            Py_RETURN_NONE;
        const Tensor out = empty({B, T, E}, kBf16, dev);
        Tensor lse;
        if (want_lse) lse = empty({B, H, T}, kF32, dev);
        const int64_t sq[3] = {T * E, D, E}, sk[3] = {S * Hkv * D, D, Hkv * D};
        const int flags = causal ? RT_MASK_CAUSAL : RT_MASK_NONE;
        void* stream = c10::cuda::getCurrentCUDAStream().stream();
        const int rc = unlocked([&] {
            return rt_attn_prefill_strided_bf16(ptr(q), ptr(k), ptr(v), ptr(&out), want_lse ? ptr<float>(&lse) : nullptr, B, H,
                                                Hkv, T, S, (int)D, sq, sk, sk, sq, flags, ptr<int32_t>(m.lens),
                                                ptr<int32_t>(m.offsets), ptr<uint8_t>(m.keep), m.keep_stride, m.scale, stream);
        });
        if (rc != RT_OK) Py_RETURN_NONE;
        return pair(out, want_lse ? &lse : nullptr);
    });
}

// q, k, v, causal, kv_lens, key_keep, scale, q_offsets
PyObject* prefill_f32(PyObject*, PyObject* const* arg, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 8) Py_RETURN_NONE;
        const Tensor *q = tensor_arg(arg[0]), *k = tensor_arg(arg[1]), *v = tensor_arg(arg[2]);
        bool causal;
        if (!q || !k || !v || !q->is_cuda() || q->dim() != 4 || k->dim() != 4 || !flag_arg(arg[3], causal)) Py_RETURN_NONE;
        const at::Device dev = q->device();
        const int64_t B = q->size(0), H = q->size(1), N = q->size(2), D = q->size(3), Hkv = k->size(1), Nkv = k->size(2);
        MaskArgs m;
        if (!dense(*q, kF32, dev) || !dense(*k, kF32, dev) || !dense(*v, kF32, dev) || k->size(0) != B || k->size(3) != D ||
            v->sizes() != k->sizes() || !mask_args(arg[4], arg[5], arg[6], arg[7], B, Nkv, dev, m))
            Py_RETURN_NONE;
        const Tensor out = empty(q->sizes(), kF32, dev), lse = empty({B, H, N}, kF32, dev);
        const int flags = causal ? RT_MASK_CAUSAL : RT_MASK_NONE;
        void* stream = c10::cuda::getCurrentCUDAStream().stream();
        const int rc = unlocked([&] {
            return rt_attn_prefill_f32(ptr<float>(q), ptr<float>(k), ptr<float>(v), ptr<float>(&out), ptr<float>(&lse), B, H,
                                       Hkv, N, Nkv, (int)D, flags, ptr<int32_t>(m.lens), ptr<int32_t>(m.offsets),
                                       ptr<uint8_t>(m.keep), m.keep_stride, m.scale, stream);
        });
        if (rc != RT_OK) Py_RETURN_NONE;
        return pair(out, &lse);
    });
}

// q, k, v, out, d_out, lse, causal, scale -> (dq, dk, dv), all f32
template <bool kIsBf16>
PyObject* backward(PyObject*, PyObject* const* arg, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 8) Py_RETURN_NONE;
        const Tensor* t[6];
        for (int i = 0; i < 6; ++i)
            if (!(t[i] = tensor_arg(arg[i]))) Py_RETURN_NONE;
        if (!t[0]->is_cuda() || t[0]->dim() != 4) Py_RETURN_NONE;
        const at::Device dev = t[0]->device();
        const int64_t B = t[0]->size(0), H = t[0]->size(1), N = t[0]->size(2), D = t[0]->size(3);
        float scale;
        bool causal;
        for (int i = 0; i < 5; ++i)
            if (!dense(*t[i], kIsBf16 ? kBf16 : kF32, dev) || t[i]->sizes() != t[0]->sizes()) Py_RETURN_NONE;
        const Tensor& lse = *t[5];
        if (!(dense(lse, kF32, dev) && lse.dim() == 3 && lse.size(0) == B && lse.size(1) == H && lse.size(2) == N) ||
            !flag_arg(arg[6], causal) || !scale_arg(arg[7], scale))
            Py_RETURN_NONE;
        const Tensor dq = empty(t[0]->sizes(), kF32, dev), dk = empty(t[0]->sizes(), kF32, dev),
                     dv = empty(t[0]->sizes(), kF32, dev);
        const size_t need = rt_attn_backward_workspace_bytes(B, H, N);
        const Tensor ws = empty({(int64_t)(need > 4 ? need : 4)}, at::kByte, dev);
        const int flags = causal ? RT_MASK_CAUSAL : RT_MASK_NONE;
        void* stream = c10::cuda::getCurrentCUDAStream().stream();
        const int rc = unlocked([&] {
            if constexpr (kIsBf16)
                return rt_attn_backward_bf16(ptr(t[0]), ptr(t[1]), ptr(t[2]), ptr(t[3]), ptr(t[4]), ptr<float>(t[5]),
                                             ptr<float>(&dq), ptr<float>(&dk), ptr<float>(&dv), B, H, N, (int)D, flags, scale,
                                             ptr(&ws), need, stream);
            else
                return rt_attn_backward_f32(ptr<float>(t[0]), ptr<float>(t[1]), ptr<float>(t[2]), ptr<float>(t[3]),
                                            ptr<float>(t[4]), ptr<float>(t[5]), ptr<float>(&dq), ptr<float>(&dk),
                                            ptr<float>(&dv), B, H, N, (int)D, flags, scale, ptr(&ws), need, stream);
        });
        if (rc != RT_OK) Py_RETURN_NONE;
        return Py_BuildValue("(NNN)", THPVariable_Wrap(dq), THPVariable_Wrap(dk), THPVariable_Wrap(dv));
    });
}

#define RT_METHOD(name, fn) {name, (PyCFunction)(void (*)(void))(fn), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {
    RT_METHOD("gqa_decode", gqa_decode),
    RT_METHOD("rope_kv_append", rope_kv_append),
    RT_METHOD("prefill_bf16", prefill_bf16),
    RT_METHOD("mha_prefill_bf16", mha_prefill_bf16),
    RT_METHOD("prefill_f32", prefill_f32),
    RT_METHOD("backward_f32", backward<false>),
    RT_METHOD("backward_bf16", backward<true>),
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_torch_binding", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__torch_binding(void) { return PyModule_Create(&kModule); }
