// Native host path of the public entry points: a CPython module over the C-ABI library.
//
// A call through ctypes costs about 20 us on the host (argument checks, output allocation, stream
// lookup and the conversion of 14-17 arguments in the interpreter), more than the GPU needs for a
// decode-sized product; here the same steps take about 4 us.  Every function takes the ordinary
// call: CUDA tensors with the layouts the kernels read.  For anything else (wrong types, operands
// that have to be copied or converted first, empty problems) it returns None and the Python function
// that called it goes through its checks, conversions and error messages.
#include <Python.h>

#include <algorithm>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/flaggems_b200.h"

namespace {

using at::ScalarType;
constexpr ScalarType E4M3 = ScalarType::Float8_e4m3fn;

// Dense CUDA tensor with storage of its own, or nullptr.
const at::Tensor* cuda_tensor(PyObject* o) {
    if (!THPVariable_Check(o)) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided) return nullptr;
    if (t.key_set().has(c10::DispatchKey::Python)) return nullptr;  // fake or wrapped tensors have no data
    return &t;
}

// C-ABI code of a bf16 / fp16 / fp32 element type, or -1.
int dtype_code(ScalarType t) {
    switch (t) {
        case ScalarType::BFloat16: return FG_DTYPE_BF16;
        case ScalarType::Half: return FG_DTYPE_F16;
        case ScalarType::Float: return FG_DTYPE_F32;
        default: return -1;
    }
}

bool py_dtype(PyObject* o, ScalarType* out) {
    if (!THPDtype_Check(o)) return false;
    *out = reinterpret_cast<THPDtype*>(o)->scalar_type;
    return true;
}

bool py_int(PyObject* o, int64_t* out) {
    if (!PyLong_Check(o)) return false;
    *out = PyLong_AsLongLong(o);
    if (*out == -1 && PyErr_Occurred()) {
        PyErr_Clear();
        return false;
    }
    return true;
}

// Truth of a Python object; false where it has none (the Python code then raises what asking for it raises).
bool py_bool(PyObject* o, bool* out) {
    const int v = PyObject_IsTrue(o);
    if (v < 0) PyErr_Clear();
    *out = v == 1;
    return v >= 0;
}

at::Tensor empty(at::IntArrayRef sizes, ScalarType dtype, const at::Tensor& like) {
    return at::Tensor(at::detail::empty_cuda(sizes, dtype, like.device(), std::nullopt));
}

void* stream_of(const at::Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// Rows of a tensor seen as [rows, last dimension]: true when one stride addresses them all.
bool as_rows(const at::Tensor& t, int64_t* rows, int64_t* cols, int64_t* ld) {
    if (t.dim() < 1 || t.numel() == 0) return false;
    *cols = t.size(-1);
    *rows = t.numel() / *cols;
    if (t.dim() == 2) {
        *ld = t.stride(0);
        return t.stride(1) == 1;
    }
    *ld = *cols;
    return t.is_contiguous();
}

// Sizes of a tensor with the last one replaced.
c10::SmallVector<int64_t, 5> sizes_with_last(const at::Tensor& t, int64_t last) {
    c10::SmallVector<int64_t, 5> s(t.sizes().begin(), t.sizes().end());
    s.back() = last;
    return s;
}

PyObject* none() { Py_RETURN_NONE; }

// The exception that _cabi.check raises for a return code.
PyObject* raise_rc(int rc) {
    const char* msg = fg_last_error();
    if (rc == FG_ERR_INVALID_ARGUMENT) {
        PyErr_SetString(PyExc_AssertionError, msg);
    } else if (rc == FG_ERR_UNSUPPORTED) {
        PyErr_SetString(PyExc_NotImplementedError, msg);
    } else {
        PyObject* mod = PyImport_ImportModule("flaggems_b200._cabi");
        PyObject* cls = mod ? PyObject_GetAttrString(mod, "FlagGemsB200Error") : nullptr;
        if (cls) PyErr_Format(cls, "flaggems_b200 error %d: %s", rc, msg);
        Py_XDECREF(cls);
        Py_XDECREF(mod);
    }
    return nullptr;
}

PyObject* pair(at::Tensor a, at::Tensor b) {
    PyObject* x = THPVariable_Wrap(std::move(a));
    PyObject* y = x ? THPVariable_Wrap(std::move(b)) : nullptr;
    if (!y) {
        Py_XDECREF(x);
        return nullptr;
    }
    PyObject* t = PyTuple_New(2);
    if (!t) {
        Py_DECREF(x);
        Py_DECREF(y);
        return nullptr;
    }
    PyTuple_SET_ITEM(t, 0, x);
    PyTuple_SET_ITEM(t, 1, y);
    return t;
}

// Runs f without the interpreter lock, as ctypes does: allocations and launches may block (a full launch queue, an
// allocation that frees cached blocks, a kernel's first load), and the thread that they wait for may be a Python one.
// The operands belong to the caller's frame, which keeps them alive.
template <typename F>
auto unlocked(F&& f) {
    struct Released {
        PyThreadState* state = PyEval_SaveThread();
        ~Released() { PyEval_RestoreThread(state); }
    } released;
    return f();
}

// C++ exceptions (an allocation that fails) become Python ones.
template <typename F>
PyObject* guarded(F&& f) {
    try {
        return f();
    } catch (const c10::OutOfMemoryError& e) {
        PyObject* torch_mod = PyImport_ImportModule("torch");
        PyObject* cls = torch_mod ? PyObject_GetAttrString(torch_mod, "OutOfMemoryError") : nullptr;
        PyErr_SetString(cls ? cls : PyExc_MemoryError, e.what_without_backtrace());
        Py_XDECREF(cls);
        Py_XDECREF(torch_mod);
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
    }
    return nullptr;
}

// ---- quantisation ---------------------------------------------------------------------------

// group_quant(x, group, eps, column_major, ue8m0) -> (q, s)
PyObject* group_quant(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        int64_t group, m, k, ld;
        if (n != 5 || !PyFloat_Check(a[2]) || !py_int(a[1], &group) || group <= 0) return none();
        const at::Tensor* x = cuda_tensor(a[0]);
        if (!x || dtype_code(x->scalar_type()) < 0 || !as_rows(*x, &m, &k, &ld) || k % group) return none();
        bool column, ue8m0;
        if (!py_bool(a[3], &column) || !py_bool(a[4], &ue8m0) || (column && x->dim() != 2)) return none();
        const float eps = (float)PyFloat_AS_DOUBLE(a[2]);
        const int64_t g = k / group;
        at::Tensor q, s;
        const int rc = unlocked([&] {
            c10::cuda::CUDAGuard guard(x->device());
            q = empty(x->sizes(), E4M3, *x);
            s = column ? at::Tensor(at::detail::empty_strided_cuda({m, g}, {1, m}, ScalarType::Float, x->device()))
                       : empty(sizes_with_last(*x, g), ScalarType::Float, *x);
            return fg_per_token_group_quant_fp8(x->data_ptr(), dtype_code(x->scalar_type()), q.data_ptr(),
                                                static_cast<float*>(s.data_ptr()), m, k, (int)group, ld, k, column ? 1 : g,
                                                column ? m : 1, eps, ue8m0, stream_of(*x));
        });
        if (rc != FG_OK) return raise_rc(rc);
        return pair(std::move(q), std::move(s));
    });
}

// act_quant(x, block, round_scales_to_powers_of_two) -> (y, s)
PyObject* act_quant(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        int64_t block, m, k, ld;
        if (n != 3 || !py_int(a[1], &block) || block <= 0) return none();
        const at::Tensor* x = cuda_tensor(a[0]);
        if (!x || x->scalar_type() != ScalarType::BFloat16 || !x->is_contiguous() || !as_rows(*x, &m, &k, &ld) || k % block)
            return none();
        bool pow2;
        if (!py_bool(a[2], &pow2)) return none();
        at::Tensor y, s;
        const int rc = unlocked([&] {
            c10::cuda::CUDAGuard guard(x->device());
            y = empty(x->sizes(), E4M3, *x);
            s = empty(sizes_with_last(*x, k / block), ScalarType::Float, *x);
            return fg_act_quant_bf16_e4m3(x->data_ptr(), y.data_ptr(), static_cast<float*>(s.data_ptr()), m, k, (int)block, k,
                                          k, k / block, pow2, stream_of(*x));
        });
        if (rc != FG_OK) return raise_rc(rc);
        return pair(std::move(y), std::move(s));
    });
}

// token_quant(x) -> (q, s): one scale per row
PyObject* token_quant(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        int64_t m, k, ld;
        const at::Tensor* x = n == 1 ? cuda_tensor(a[0]) : nullptr;
        if (!x || dtype_code(x->scalar_type()) < 0 || !as_rows(*x, &m, &k, &ld)) return none();
        at::Tensor q, s;
        const int rc = unlocked([&] {
            c10::cuda::CUDAGuard guard(x->device());
            q = empty(x->sizes(), E4M3, *x);
            s = empty(sizes_with_last(*x, 1), ScalarType::Float, *x);
            return fg_per_token_quant_fp8(x->data_ptr(), dtype_code(x->scalar_type()), q.data_ptr(),
                                          static_cast<float*>(s.data_ptr()), m, k, ld, k, nullptr, 1, 0, nullptr, stream_of(*x));
        });
        if (rc != FG_OK) return raise_rc(rc);
        return pair(std::move(q), std::move(s));
    });
}

// tensor_quant(x, scale) -> q: the given scale for the whole tensor
PyObject* tensor_quant(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        int64_t m, k, ld;
        const at::Tensor* x = n == 2 ? cuda_tensor(a[0]) : nullptr;
        const at::Tensor* s = x ? cuda_tensor(a[1]) : nullptr;
        if (!s || s->scalar_type() != ScalarType::Float || s->numel() < 1 || dtype_code(x->scalar_type()) < 0 ||
            !as_rows(*x, &m, &k, &ld))
            return none();
        at::Tensor q;
        const int rc = unlocked([&] {
            c10::cuda::CUDAGuard guard(x->device());
            q = empty(x->sizes(), E4M3, *x);
            float* scale = static_cast<float*>(s->data_ptr());
            return fg_per_tensor_quant_fp8(x->data_ptr(), dtype_code(x->scalar_type()), q.data_ptr(), scale, 0, scale, m, k, ld,
                                           k, nullptr, 1, 0, nullptr, stream_of(*x));
        });
        if (rc != FG_OK) return raise_rc(rc);
        return THPVariable_Wrap(std::move(q));
    });
}

// ---- products -------------------------------------------------------------------------------

// [K, N] operand in column-major storage with 16-byte aligned columns (TMA reads it as rows of N).
bool k_contiguous(const at::Tensor& b) { return b.stride(0) == 1 && b.stride(1) % 16 == 0; }

// block_mm(A, B, As, Bs, [128, 128], output dtype) -> C
PyObject* block_mm(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        ScalarType out;
        int64_t bn, bk, m, k, ld;
        if (n != 6 || !PyList_Check(a[4]) || PyList_GET_SIZE(a[4]) != 2 || !py_int(PyList_GET_ITEM(a[4], 0), &bn) ||
            !py_int(PyList_GET_ITEM(a[4], 1), &bk) || bn != 128 || bk != 128 || !py_dtype(a[5], &out) || dtype_code(out) < 0)
            return none();
        const at::Tensor *A = cuda_tensor(a[0]), *B = cuda_tensor(a[1]), *As = cuda_tensor(a[2]), *Bs = cuda_tensor(a[3]);
        if (!A || !B || !As || !Bs || A->scalar_type() != E4M3 || B->scalar_type() != E4M3 ||
            As->scalar_type() != ScalarType::Float || Bs->scalar_type() != ScalarType::Float)
            return none();
        if (!A->is_contiguous() || !as_rows(*A, &m, &k, &ld) || B->dim() != 2 || Bs->dim() != 2 || B->size(1) != k) return none();
        const int64_t rows_b = B->size(0), kb = (k + 127) / 128;
        if (rows_b == 0 || B->stride(1) != 1 || B->stride(0) % 16 || Bs->size(0) != (rows_b + 127) / 128 || Bs->size(1) != kb)
            return none();
        if (As->dim() != A->dim() || As->size(-1) != kb) return none();
        for (int64_t d = 0; d + 1 < A->dim(); ++d)
            if (As->size(d) != A->size(d)) return none();
        int64_t as_row = kb, as_col = 1;
        if (As->dim() == 2) {
            as_row = As->stride(0);
            as_col = As->stride(1);
        } else if (!As->is_contiguous()) {
            return none();
        }
        at::Tensor c;
        const int rc = unlocked([&] {
            c10::cuda::CUDAGuard guard(A->device());
            c = empty(sizes_with_last(*A, rows_b), out, *A);
            return fg_block_scaled_mm_fp8(c.data_ptr(), A->data_ptr(), B->data_ptr(), static_cast<const float*>(As->data_ptr()),
                                          static_cast<const float*>(Bs->data_ptr()), m, rows_b, k, k, B->stride(0), rows_b,
                                          as_row, as_col, Bs->stride(0), Bs->stride(1), dtype_code(out), stream_of(*A));
        });
        if (rc != FG_OK) return raise_rc(rc);
        return THPVariable_Wrap(std::move(c));
    });
}

bool scale_ok(const at::Tensor& s, int64_t full) {
    return s.scalar_type() == ScalarType::Float && s.is_contiguous() && (s.numel() == 1 || s.numel() == full);
}

// scaled_mm(c, a, b, a_scale, b_scale, bias or None, cutlass) -> c.  ``cutlass`` selects the rules of
// cutlass_scaled_mm (aligned rows of c, scales of any shape with M / N values, the bias added after
// rounding); otherwise those of aten _scaled_mm (scales [M] or [M, 1] and [N] or [1, N]).
PyObject* scaled_mm(PyObject*, PyObject* const* p, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 7) return none();
        const at::Tensor *c = cuda_tensor(p[0]), *a = cuda_tensor(p[1]), *b = cuda_tensor(p[2]), *sa = cuda_tensor(p[3]),
                         *sb = cuda_tensor(p[4]);
        if (!c || !a || !b || !sa || !sb || a->scalar_type() != E4M3 || b->scalar_type() != E4M3) return none();
        if (a->dim() != 2 || b->dim() != 2 || c->dim() != 2) return none();
        const int64_t m = a->size(0), k = a->size(1), cols = b->size(1);
        const int code = c->scalar_type() == E4M3 ? FG_DTYPE_E4M3 : dtype_code(c->scalar_type());
        if (code < 0 || m == 0 || cols == 0 || b->size(0) != k || c->size(0) != m || c->size(1) != cols) return none();
        if (a->stride(1) != 1 || a->stride(0) % 16 || c->stride(1) != 1 || !k_contiguous(*b)) return none();
        if (!scale_ok(*sa, m) || !scale_ok(*sb, cols)) return none();
        const bool cutlass = p[6] == Py_True;
        if (cutlass) {
            if (c->stride(0) % 16 || code == FG_DTYPE_E4M3) return none();
        } else {
            if (sa->numel() > 1 && !(sa->dim() == 1 || (sa->dim() == 2 && sa->size(1) == 1))) return none();
            if (sb->numel() > 1 && !(sb->dim() == 1 || (sb->dim() == 2 && sb->size(0) == 1))) return none();
        }
        const at::Tensor* bias = nullptr;
        if (p[5] != Py_None) {
            bias = cuda_tensor(p[5]);
            const ScalarType want = code == FG_DTYPE_E4M3 ? ScalarType::Float : c->scalar_type();
            if (!bias || bias->scalar_type() != want || bias->dim() != 1 || bias->size(0) != cols || !bias->is_contiguous()) return none();
        }
        const int rc = unlocked([&] {
            c10::cuda::CUDAGuard guard(a->device());
            return fg_scaled_mm_fp8(c->data_ptr(), a->data_ptr(), b->data_ptr(), static_cast<const float*>(sa->data_ptr()),
                                    static_cast<const float*>(sb->data_ptr()), bias ? bias->data_ptr() : nullptr, m, cols, k,
                                    a->stride(0), b->stride(1), c->stride(0), sa->numel() > 1 ? FG_SCALE_VECTOR : FG_SCALE_SCALAR,
                                    sb->numel() > 1 ? FG_SCALE_VECTOR : FG_SCALE_SCALAR, code, cutlass, stream_of(*a));
        });
        if (rc != FG_OK) return raise_rc(rc);
        Py_INCREF(p[0]);
        return p[0];
    });
}

// scaled_mm_new(a, b, a_scale, b_scale, bias or None, output dtype) -> C
PyObject* scaled_mm_new(PyObject* self, PyObject* const* p, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        ScalarType out;
        const at::Tensor *a = n == 6 ? cuda_tensor(p[0]) : nullptr, *b = a ? cuda_tensor(p[1]) : nullptr;
        if (!b || a->dim() != 2 || b->dim() != 2 || !py_dtype(p[5], &out) || (out != E4M3 && dtype_code(out) < 0)) return none();
        if (a->size(0) == 0 || b->size(1) == 0) return none();
        PyObject* c = THPVariable_Wrap(unlocked([&] { return empty({a->size(0), b->size(1)}, out, *a); }));
        if (!c) return nullptr;
        PyObject* args[7] = {c, p[0], p[1], p[2], p[3], p[4], Py_False};
        PyObject* r = scaled_mm(self, args, 7);
        Py_DECREF(c);
        return r;
    });
}

// grouped_mm(a, b, scale_a, scale_b, offs, output dtype) -> C: rows of a [M, K] grouped by offs, b [G, K, N]
PyObject* grouped_mm(PyObject*, PyObject* const* p, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        ScalarType out;
        if (n != 6 || !py_dtype(p[5], &out) || dtype_code(out) < 0) return none();
        const at::Tensor *a = cuda_tensor(p[0]), *b = cuda_tensor(p[1]), *sa = cuda_tensor(p[2]), *sb = cuda_tensor(p[3]),
                         *offs = cuda_tensor(p[4]);
        if (!a || !b || !sa || !sb || !offs || a->scalar_type() != E4M3 || b->scalar_type() != E4M3) return none();
        if (a->dim() != 2 || b->dim() != 3 || sa->dim() != 1 || sb->dim() != 2 || offs->dim() != 1) return none();
        const int64_t m = a->size(0), k = a->size(1), groups = b->size(0), cols = b->size(2);
        if (m == 0 || cols == 0 || groups == 0 || k == 0 || k % 16 || b->size(1) != k) return none();
        if (b->stride(1) != 1 || b->stride(2) != k || (groups > 1 && b->stride(0) != k * cols)) return none();
        if (a->stride(1) != 1 || a->stride(0) % 16 || (uintptr_t)a->data_ptr() % 16) return none();
        if (sa->scalar_type() != ScalarType::Float || sa->size(0) != m || !sa->is_contiguous() ||
            sb->scalar_type() != ScalarType::Float || sb->size(0) != groups || sb->size(1) != cols || !sb->is_contiguous() ||
            offs->scalar_type() != ScalarType::Int || offs->size(0) != groups || !offs->is_contiguous())
            return none();
        at::Tensor c, ws;
        const int rc = unlocked([&] {
            c10::cuda::CUDAGuard guard(a->device());
            c = empty({m, cols}, out, *a);
            const int64_t need = fg_scaled_grouped_mm_workspace_bytes(m, (int)groups, k) + 256;
            ws = empty({need}, ScalarType::Byte, *a);
            return fg_scaled_grouped_mm_fp8(c.data_ptr(), a->data_ptr(), b->data_ptr(), static_cast<const float*>(sa->data_ptr()),
                                            static_cast<const float*>(sb->data_ptr()), nullptr, 0,
                                            static_cast<const int32_t*>(offs->data_ptr()), (int)groups, m, cols, k, a->stride(0),
                                            cols, dtype_code(out), ws.data_ptr(), need, stream_of(*a));
        });
        if (rc != FG_OK) return raise_rc(rc);
        return THPVariable_Wrap(std::move(c));
    });
}

// ---- routing and MoE glue -----------------------------------------------------------------------

// topk_softmax(weights, indices, source_rows, gating, renormalize) -> True
PyObject* topk_softmax(PyObject*, PyObject* const* p, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 5) return none();
        const at::Tensor *w = cuda_tensor(p[0]), *idx = cuda_tensor(p[1]), *src = cuda_tensor(p[2]), *g = cuda_tensor(p[3]);
        if (!w || !idx || !src || !g || g->dim() != 2 || w->dim() != 2) return none();
        const int64_t t = g->size(0), e = g->size(1), k = w->size(1);
        if (t == 0 || k > 32 || w->scalar_type() != ScalarType::Float || src->scalar_type() != ScalarType::Int) return none();
        if (w->size(0) != t || idx->sizes() != w->sizes() || src->sizes() != w->sizes()) return none();
        if (!w->is_contiguous() || !idx->is_contiguous() || !src->is_contiguous() || !g->is_contiguous()) return none();
        const ScalarType it = idx->scalar_type();
        const int kind = it == ScalarType::Int ? 0 : it == ScalarType::UInt32 ? 1 : it == ScalarType::Long ? 2 : -1;
        if (kind < 0 || dtype_code(g->scalar_type()) < 0) return none();
        bool renormalize;
        if (!py_bool(p[4], &renormalize)) return none();
        const int rc = unlocked([&] {
            c10::cuda::CUDAGuard guard(g->device());
            return fg_topk_softmax(static_cast<float*>(w->data_ptr()), idx->data_ptr(), kind, static_cast<int32_t*>(src->data_ptr()),
                                   g->data_ptr(), dtype_code(g->scalar_type()), t, (int)e, (int)k, renormalize, nullptr,
                                   stream_of(*g));
        });
        if (rc != FG_OK) return raise_rc(rc);
        Py_RETURN_TRUE;
    });
}

// grouped_topk(scores, n_group, topk_group, topk, renormalize, scaling, bias, scoring_func) -> (weights, indices)
PyObject* grouped_topk(PyObject*, PyObject* const* p, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        int64_t n_group, topk_group, topk, scoring;
        if (n != 8 || !py_int(p[1], &n_group) || !py_int(p[2], &topk_group) || !py_int(p[3], &topk) || !py_int(p[7], &scoring) ||
            !PyFloat_Check(p[5]))
            return none();
        const at::Tensor *s = cuda_tensor(p[0]), *bias = cuda_tensor(p[6]);
        if (!s || !bias || s->dim() != 2 || bias->dim() != 1 || dtype_code(s->scalar_type()) < 0) return none();
        const int64_t t = s->size(0), e = s->size(1);
        if (t == 0 || n_group < 1 || n_group > 32 || e % n_group || topk > 32 || (scoring != 0 && scoring != 1)) return none();
        if (s->stride(1) != 1 || bias->scalar_type() != s->scalar_type() || bias->size(0) != e || !bias->is_contiguous())
            return none();
        bool renormalize;
        if (!py_bool(p[4], &renormalize)) return none();
        const float scaling = (float)PyFloat_AS_DOUBLE(p[5]);
        at::Tensor w, idx;
        const int rc = unlocked([&] {
            c10::cuda::CUDAGuard guard(s->device());
            w = empty({t, topk}, ScalarType::Float, *s);
            idx = empty({t, topk}, ScalarType::Int, *s);
            return fg_grouped_topk(static_cast<float*>(w.data_ptr()), static_cast<int32_t*>(idx.data_ptr()), s->data_ptr(),
                                   bias->data_ptr(), dtype_code(s->scalar_type()), t, (int)e, s->stride(0), (int)n_group,
                                   (int)topk_group, (int)topk, renormalize, scaling, (int)scoring, nullptr, stream_of(*s));
        });
        if (rc != FG_OK) return raise_rc(rc);
        return pair(std::move(w), std::move(idx));
    });
}

// moe_align(topk_ids, block_size, num_experts, length of sorted_ids) -> (sorted_ids, expert_ids, num_tokens_post_pad)
PyObject* moe_align(PyObject*, PyObject* const* p, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        int64_t bs, e, pad;
        const at::Tensor* ids = n == 4 ? cuda_tensor(p[0]) : nullptr;
        if (!ids || !py_int(p[1], &bs) || !py_int(p[2], &e) || !py_int(p[3], &pad) || bs <= 0 || !ids->is_contiguous())
            return none();
        const bool i64 = ids->scalar_type() == ScalarType::Long;
        if (!i64 && ids->scalar_type() != ScalarType::Int) return none();
        at::Tensor sorted, eids, post;
        const int rc = unlocked([&] {
            c10::cuda::CUDAGuard guard(ids->device());
            sorted = empty({pad}, ScalarType::Int, *ids);
            eids = empty({(pad + bs - 1) / bs}, ScalarType::Int, *ids);
            post = empty({1}, ScalarType::Int, *ids);
            return fg_moe_align_block_size(ids->data_ptr(), i64, ids->numel(), (int)e, (int)bs, nullptr, 0,
                                           static_cast<int32_t*>(sorted.data_ptr()), pad, static_cast<int32_t*>(eids.data_ptr()),
                                           eids.numel(), static_cast<int32_t*>(post.data_ptr()), stream_of(*ids));
        });
        if (rc != FG_OK) return raise_rc(rc);
        PyObject* t = PyTuple_New(3);
        if (!t) return nullptr;
        at::Tensor* out[3] = {&sorted, &eids, &post};
        for (int i = 0; i < 3; ++i) {
            PyObject* o = THPVariable_Wrap(std::move(*out[i]));
            if (!o) {
                Py_DECREF(t);
                return nullptr;
            }
            PyTuple_SET_ITEM(t, i, o);
        }
        return t;
    });
}

// silu_mul(a, b, out or None) -> out
PyObject* silu_mul(PyObject*, PyObject* const* p, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        const at::Tensor *x = n == 3 ? cuda_tensor(p[0]) : nullptr, *y = x ? cuda_tensor(p[1]) : nullptr;
        int64_t m, k, ldx, ldy, ldo, m2, k2;
        if (!y || x->sizes() != y->sizes() || x->scalar_type() != y->scalar_type() || dtype_code(x->scalar_type()) < 0)
            return none();
        if (!as_rows(*x, &m, &k, &ldx) || !as_rows(*y, &m2, &k2, &ldy)) return none();
        at::Tensor made;
        const at::Tensor* o = nullptr;
        if (p[2] == Py_None) {
            made = unlocked([&] { return empty(x->sizes(), x->scalar_type(), *x); });
            o = &made;
        } else {
            o = cuda_tensor(p[2]);
            if (!o || o->sizes() != x->sizes() || o->scalar_type() != x->scalar_type()) return none();
        }
        if (!as_rows(*o, &m2, &k2, &ldo)) return none();
        const int rc = unlocked([&] {
            c10::cuda::CUDAGuard guard(x->device());
            return fg_silu_and_mul(x->data_ptr(), y->data_ptr(), o->data_ptr(), m, k, ldx, ldy, ldo, dtype_code(x->scalar_type()),
                                   stream_of(*x));
        });
        if (rc != FG_OK) return raise_rc(rc);
        if (made.defined()) return THPVariable_Wrap(std::move(made));
        Py_INCREF(p[2]);
        return p[2];
    });
}

// moe_sum(input [M, topk, K], output [M, K]) -> output
PyObject* moe_sum(PyObject*, PyObject* const* p, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        const at::Tensor *x = n == 2 ? cuda_tensor(p[0]) : nullptr, *o = x ? cuda_tensor(p[1]) : nullptr;
        if (!o || x->dim() != 3 || o->dim() != 2 || x->scalar_type() != o->scalar_type() || dtype_code(x->scalar_type()) < 0)
            return none();
        if (o->size(0) != x->size(0) || o->size(1) != x->size(2) || !x->is_contiguous() || !o->is_contiguous()) return none();
        const int rc = unlocked([&] {
            c10::cuda::CUDAGuard guard(x->device());
            return fg_moe_sum(x->data_ptr(), o->data_ptr(), x->size(0), (int)x->size(1), x->size(2), dtype_code(x->scalar_type()),
                              stream_of(*x));
        });
        if (rc != FG_OK) return raise_rc(rc);
        Py_INCREF(p[1]);
        return p[1];
    });
}

// fused_experts(hidden, w1, w2, topk_weights, topk_ids, out, mode, w1_scale, w2_scale, a1_scale, a2_scale,
//               num_experts, expert_map, tokens per chunk) -> out.  The caller has checked shapes, types and
// layouts; scales, map and the two activation scales may be None.
PyObject* fused_experts(PyObject*, PyObject* const* p, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        int64_t mode, experts, chunk;
        if (n != 14 || !py_int(p[6], &mode) || !py_int(p[11], &experts) || !py_int(p[13], &chunk)) return none();
        const at::Tensor *x = cuda_tensor(p[0]), *w1 = cuda_tensor(p[1]), *w2 = cuda_tensor(p[2]), *tw = cuda_tensor(p[3]),
                         *ids = cuda_tensor(p[4]), *out = cuda_tensor(p[5]);
        if (!x || !w1 || !w2 || !tw || !ids || !out) return none();
        const float* f[4] = {nullptr, nullptr, nullptr, nullptr};
        for (int i = 0; i < 4; ++i) {
            if (p[7 + i] == Py_None) continue;
            const at::Tensor* s = cuda_tensor(p[7 + i]);
            if (!s || s->scalar_type() != ScalarType::Float) return none();
            f[i] = static_cast<const float*>(s->data_ptr());
        }
        const at::Tensor* map = nullptr;
        if (p[12] != Py_None && !(map = cuda_tensor(p[12]))) return none();
        const int64_t t = x->size(0), h = x->size(1), inter = w2->size(2), topk = ids->size(1);
        const int code = dtype_code(x->scalar_type()), esz = (int)x->element_size();
        const bool i64 = ids->scalar_type() == ScalarType::Long;
        at::Tensor ws;
        const int rc = unlocked([&] {
            c10::cuda::CUDAGuard guard(x->device());
            const int64_t most = t < chunk ? t : chunk;
            const int64_t need = fg_fused_experts_workspace_bytes(
                (int)mode, most, (int)topk, (int)std::max(experts, w1->size(0)), h, inter, code);
            ws = empty({need}, ScalarType::Byte, *x);
            for (int64_t b = 0; b < t; b += chunk) {
                const int64_t rows = t - b < chunk ? t - b : chunk;
                const int e = fg_fused_experts(
                    static_cast<char*>(out->data_ptr()) + b * h * esz, static_cast<const char*>(x->data_ptr()) + b * h * esz, code,
                    static_cast<const char*>(ids->data_ptr()) + b * topk * (i64 ? 8 : 4), i64,
                    static_cast<const char*>(tw->data_ptr()) + b * topk * tw->element_size(), dtype_code(tw->scalar_type()), rows,
                    (int)topk, w1->data_ptr(), w2->data_ptr(), f[0], f[1], f[2], f[3], (int)mode, (int)experts, (int)w1->size(0),
                    map ? static_cast<const int32_t*>(map->data_ptr()) : nullptr, map ? (int)map->numel() : 0, h, inter, nullptr,
                    ws.data_ptr(), need, stream_of(*x));
                if (e != FG_OK) return e;
            }
            return (int)FG_OK;
        });
        if (rc != FG_OK) return raise_rc(rc);
        Py_INCREF(p[5]);
        return p[5];
    });
}

#define FG_METHOD(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    FG_METHOD(group_quant), FG_METHOD(act_quant),    FG_METHOD(token_quant), FG_METHOD(tensor_quant),
    FG_METHOD(block_mm),    FG_METHOD(scaled_mm),    FG_METHOD(scaled_mm_new), FG_METHOD(grouped_mm),
    FG_METHOD(topk_softmax), FG_METHOD(grouped_topk), FG_METHOD(moe_align),  FG_METHOD(silu_mul),
    FG_METHOD(moe_sum),     FG_METHOD(fused_experts), {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fg_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fg_host(void) { return PyModule_Create(&module); }
