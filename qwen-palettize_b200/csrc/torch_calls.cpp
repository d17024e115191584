// Python module _plz_torch: the calls that a program makes once per Linear (plz_ops.py), each as one C++ call. From Python an operation of one launch costs 15 to
// 20 us of host time, 3.6 of them the launch: descriptors built field by field, ctypes conversions, torch.empty, the stream looked up. A token's Linear (8 us of
// GPU time) and the reference's functions under autograd wait for that.
//
// Every function here takes plain CUDA tensors that fit together and returns None for everything else, and where the library refuses the call; the caller then takes
// its general path, which raises what it always raised. Nothing is kept between calls. The interpreter's lock is given up while the library launches.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/plz.h"

namespace {

// an exact torch.Tensor or Parameter on a GPU with memory of its own (under vmap and jvp there are some without), or nullptr
const at::Tensor* tensor(PyObject* o) {
    if (!THPVariable_CheckExact(o)) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(o);
    return t.defined() && t.is_cuda() && t.layout() == at::kStrided && t.has_storage() ? &t : nullptr;
}
const at::Tensor* matrix(PyObject* o, int64_t cols = -1) {
    const at::Tensor* t = tensor(o);
    return t && t->scalar_type() == at::kBFloat16 && t->dim() == 2 && t->stride(1) == 1 && (cols < 0 || t->size(1) == cols) ? t : nullptr;
}
bool whole(PyObject* o, int64_t& v) {
    if (!PyLong_CheckExact(o)) return false;
    v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
    return true;
}
bool real(PyObject* o, double& v) {
    if (PyFloat_CheckExact(o)) { v = PyFloat_AS_DOUBLE(o); return true; }
    int64_t i;
    if (!whole(o, i)) return false;
    v = (double)i;
    return true;
}
bool truth(PyObject* o, bool& v) {
    v = o == Py_True;
    return o == Py_True || o == Py_False;
}

constexpr int kWeightArgs = 6;   // packed, palette, N, K, gs_n, gs_k
bool weight(PyObject* const* a, plz_weight_t& w) {
    const at::Tensor *packed = tensor(a[0]), *palette = tensor(a[1]);
    int64_t v[4];
    for (int i = 0; i < 4; ++i)
        if (!whole(a[2 + i], v[i]) || v[i] <= 0 || v[i] > 0x7FFFFFFF) return false;
    if (!packed || !palette || packed->scalar_type() != at::kByte || packed->dim() != 2 || packed->stride(1) != 1) return false;
    if (palette->scalar_type() != at::kBFloat16 || !palette->is_contiguous() || palette->numel() != (v[0] / v[2]) * (v[1] / v[3]) * 4) return false;
    w = {(int32_t)v[0], (int32_t)v[1], (int32_t)v[2], (int32_t)v[3], packed->data_ptr(), packed->stride(0), palette->data_ptr()};
    return true;
}
int64_t palette_groups(const plz_weight_t& w) { return (int64_t)(w.N / w.gs_n) * (w.K / w.gs_k); }
bool rows(const at::Tensor& t) { return t.size(0) <= 0x7FFFFFFF; }
struct Rows { void* p; int64_t ld; int32_t n; };
Rows rows_of(const at::Tensor& t) { return {t.data_ptr(), t.stride(0), (int32_t)t.size(0)}; }
at::Tensor result(const at::Tensor& like, at::IntArrayRef sizes, at::ScalarType type = at::kBFloat16) { return at::empty(sizes, like.options().dtype(type)); }

// gives the interpreter's lock up for its lifetime; an exception takes it back too
struct Unlocked {
    PyThreadState* state = PyEval_SaveThread();
    ~Unlocked() { PyEval_RestoreThread(state); }
};
// call: addresses and library calls only, tensors are looked at before
template <typename F>
bool launch(F call) {
    void* stream = c10::cuda::getCurrentCUDAStream().stream();
    Unlocked unlocked;
    return call(stream) == PLZ_OK;
}
bool clear(void* p, int64_t words, void* stream) {   // fp32
    const int64_t bytes = words * 4;
    return plz_zero(&p, &bytes, 1, stream) == PLZ_OK;
}

// (weight, x) -> y
PyObject* hard_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    plz_weight_t w;
    const at::Tensor* x;
    if (n != kWeightArgs + 1 || !weight(a, w) || !(x = matrix(a[6], w.K)) || !rows(*x)) Py_RETURN_NONE;
    at::Tensor y = result(*x, {x->size(0), w.N});
    const Rows xr = rows_of(*x), yr = rows_of(y);
    if (!launch([&](void* s) { return plz_hard_fwd(&w, xr.p, xr.ld, xr.n, nullptr, nullptr, yr.p, w.N, s); })) Py_RETURN_NONE;
    return THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

// (weight, x) -> y for up to 64 rows
PyObject* hard_forward_smallm(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    plz_weight_t w;
    const at::Tensor* x;
    if (n != kWeightArgs + 1 || !weight(a, w) || !(x = matrix(a[6], w.K)) || x->size(0) > 64) Py_RETURN_NONE;
    at::Tensor y = result(*x, {x->size(0), w.N});
    const Rows xr = rows_of(*x), yr = rows_of(y);
    if (!launch([&](void* s) { return plz_hard_fwd_smallm(&w, xr.p, xr.ld, xr.n, yr.p, w.N, s); })) Py_RETURN_NONE;
    return THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

// (weight, x, bias or None) -> y
PyObject* hard_forward_bias(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    plz_weight_t w;
    const at::Tensor *x, *bias = nullptr;
    if (n != kWeightArgs + 2 || !weight(a, w) || !(x = matrix(a[6], w.K)) || !rows(*x)) Py_RETURN_NONE;
    if (a[7] != Py_None && (!(bias = tensor(a[7])) || bias->scalar_type() != at::kBFloat16 || !bias->is_contiguous() || bias->numel() != w.N)) Py_RETURN_NONE;
    at::Tensor y = result(*x, {x->size(0), w.N});
    const Rows xr = rows_of(*x), yr = rows_of(y);
    const void* bp = bias ? bias->data_ptr() : nullptr;
    if (!launch([&](void* s) { return plz_hard_fwd_bias(&w, xr.p, xr.ld, xr.n, bp, yr.p, w.N, s); })) Py_RETURN_NONE;
    return THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

// (weight, x, A or None, B, scale) -> y of x's shape with N columns: what a Linear in eval mode does
PyObject* eval_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    plz_weight_t w;
    const at::Tensor* x;
    plz_lora_t lora = {};
    if (n != kWeightArgs + 4 || !weight(a, w) || !(x = tensor(a[6]))) Py_RETURN_NONE;
    if (x->scalar_type() != at::kBFloat16 || x->dim() < 1 || x->size(-1) != w.K || !x->is_contiguous() || x->numel() == 0) Py_RETURN_NONE;
    const int64_t M = x->numel() / w.K;
    if (M > 0x7FFFFFFF) Py_RETURN_NONE;
    at::DimVector shape(x->sizes().begin(), x->sizes().end());
    shape.back() = w.N;
    at::Tensor t;
    if (a[7] != Py_None) {
        const at::Tensor *A = matrix(a[7], w.K), *B = matrix(a[8]);
        double scale;
        if (!A || !B || A->size(0) != B->size(1) || A->size(0) < 1 || A->size(0) > 64 || B->size(0) != w.N || !real(a[9], scale)) Py_RETURN_NONE;
        lora = {(int32_t)A->size(0), (float)scale, A->data_ptr(), A->stride(0), B->data_ptr(), B->stride(0)};
        t = result(*x, {M, A->size(0)});
    }
    at::Tensor y = result(*x, shape);
    const bool with_lora = t.defined();
    void *const xp = x->data_ptr(), *const yp = y.data_ptr(), *const tp = with_lora ? t.data_ptr() : nullptr;
    if (!launch([&](void* s) {
            if (!with_lora && M <= 64) return plz_hard_fwd_smallm(&w, xp, w.K, (int32_t)M, yp, w.N, s);
            return plz_hard_fwd(&w, xp, w.K, (int32_t)M, with_lora ? &lora : nullptr, tp, yp, w.N, s);
        }))
        Py_RETURN_NONE;
    return THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

// (weight, dy) -> dx
PyObject* backward_dx(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    plz_weight_t w;
    const at::Tensor* dy;
    if (n != kWeightArgs + 1 || !weight(a, w) || !(dy = matrix(a[6], w.N)) || !rows(*dy)) Py_RETURN_NONE;
    at::Tensor dx = result(*dy, {dy->size(0), w.K});
    const Rows dyr = rows_of(*dy), dxr = rows_of(dx);
    if (!launch([&](void* s) { return plz_bwd_dx(&w, dyr.p, dyr.ld, dyr.n, nullptr, nullptr, dxr.p, w.K, s); })) Py_RETURN_NONE;
    return THPVariable_Wrap(std::move(dx));
    END_HANDLE_TH_ERRORS
}

// (weight, x, dy) -> dpalette
PyObject* backward_dw_hard(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    plz_weight_t w;
    const at::Tensor *x, *dy;
    if (n != kWeightArgs + 2 || !weight(a, w) || !(x = matrix(a[6], w.K)) || !(dy = matrix(a[7], w.N)) || !rows(*x) || dy->size(0) != x->size(0)) Py_RETURN_NONE;
    at::Tensor dpal = result(*x, {palette_groups(w), 4}, at::kFloat);
    const Rows xr = rows_of(*x), dyr = rows_of(*dy);
    float* const pp = (float*)dpal.data_ptr();
    const int64_t words = dpal.numel();
    if (!launch([&](void* s) {
            if (!clear(pp, words, s)) return PLZ_ERR_CUDA;
            return plz_bwd_dw_hard(&w, xr.p, xr.ld, dyr.p, dyr.ld, xr.n, pp, s);
        }))
        Py_RETURN_NONE;
    return THPVariable_Wrap(std::move(dpal));
    END_HANDLE_TH_ERRORS
}

// (dy) -> sums of its columns
PyObject* col_sum(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    const at::Tensor* dy;
    if (n != 1 || !(dy = matrix(a[0])) || !rows(*dy) || dy->size(1) > 0x7FFFFFFF) Py_RETURN_NONE;
    at::Tensor out = result(*dy, {dy->size(1)}, at::kFloat);
    const Rows dyr = rows_of(*dy);
    const int64_t cols = dy->size(1);
    float* const sums = (float*)out.data_ptr();
    if (!launch([&](void* s) {
            if (!clear(sums, cols, s)) return PLZ_ERR_CUDA;
            return plz_col_sum(dyr.p, dyr.ld, dyr.n, (int32_t)cols, sums, s);
        }))
        Py_RETURN_NONE;
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// planar: (4, K, N), else [N, K, 4]
bool logits_of(PyObject* o, bool planar, plz_logits_t& l, const at::Tensor*& t) {
    t = tensor(o);
    if (!t || t->dim() != 3 || (t->scalar_type() != at::kFloat && t->scalar_type() != at::kHalf)) return false;
    l = {t->data_ptr(), t->scalar_type() == at::kHalf, planar ? t->stride(2) : t->stride(0), t->stride(1), planar ? t->stride(0) : t->stride(2)};
    return true;
}
bool noise_of(PyObject* o, bool planar, int64_t seed, plz_noise_t& z) {
    z = {};
    if (o == Py_None) return true;
    if (PyUnicode_Check(o)) { z.mode = 2; z.seed = (uint32_t)seed; return true; }
    const at::Tensor* t = tensor(o);
    if (!t || t->dim() != 3 || t->scalar_type() != at::kFloat) return false;
    z = {1, 0, (const float*)t->data_ptr(), planar ? t->stride(2) : t->stride(0), t->stride(1), planar ? t->stride(0) : t->stride(2)};
    return true;
}

// (weight, logits, planar, noise, tau): the hard indices into the weight's packed rows -> True. They do not depend on the noise, whose type is looked at all the same.
PyObject* select_indices(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    plz_weight_t w;
    plz_logits_t l;
    plz_noise_t z;
    const at::Tensor* t;
    bool planar;
    double tau;
    if (n != kWeightArgs + 4 || !weight(a, w) || !truth(a[7], planar) || !logits_of(a[6], planar, l, t) || !noise_of(a[8], planar, 0, z) || !real(a[9], tau)) Py_RETURN_NONE;
    if (!launch([&](void* s) { return plz_soft_select(&w, &l, nullptr, (float)tau, 1, nullptr, w.K, 1, s); })) Py_RETURN_NONE;
    Py_RETURN_TRUE;
    END_HANDLE_TH_ERRORS
}

// (weight, x, dy, logits, planar, noise, tau, seed, want dlogits, want dpalette) -> (dlogits or None, dpalette or None)
PyObject* backward_dw_soft(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    plz_weight_t w;
    plz_logits_t l;
    plz_noise_t z;
    const at::Tensor *x, *dy, *t;
    bool planar, want_l, want_p;
    double tau;
    int64_t seed;
    if (n != kWeightArgs + 9 || !weight(a, w) || !(x = matrix(a[6], w.K)) || !(dy = matrix(a[7], w.N)) || !rows(*x) || dy->size(0) != x->size(0)) Py_RETURN_NONE;
    if (!truth(a[9], planar) || !logits_of(a[8], planar, l, t) || !real(a[11], tau) || !whole(a[12], seed) || !noise_of(a[10], planar, seed, z)) Py_RETURN_NONE;
    if (!truth(a[13], want_l) || !truth(a[14], want_p)) Py_RETURN_NONE;
    at::Tensor dlog, dpal;
    if (want_l) {
        dlog = at::empty_like(*t);
        if (dlog.strides() != t->strides()) Py_RETURN_NONE;
    }
    if (want_p) dpal = result(*x, {palette_groups(w), 4}, at::kFloat);
    const Rows xr = rows_of(*x), dyr = rows_of(*dy);
    void* const lp = want_l ? dlog.data_ptr() : nullptr;
    float* const pp = want_p ? (float*)dpal.data_ptr() : nullptr;
    const int64_t words = want_p ? dpal.numel() : 0;
    if (!launch([&](void* s) {
            if (want_p && !clear(pp, words, s)) return PLZ_ERR_CUDA;
            return plz_bwd_dw_soft(&w, xr.p, xr.ld, dyr.p, dyr.ld, xr.n, &l, &z, (float)tau, lp, pp, s);
        }))
        Py_RETURN_NONE;
    PyObject* out = PyTuple_New(2);
    if (!out) return nullptr;
    PyTuple_SET_ITEM(out, 0, want_l ? THPVariable_Wrap(std::move(dlog)) : Py_NewRef(Py_None));
    PyTuple_SET_ITEM(out, 1, want_p ? THPVariable_Wrap(std::move(dpal)) : Py_NewRef(Py_None));
    return out;
    END_HANDLE_TH_ERRORS
}

#define PLZ_CALL(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {PLZ_CALL(hard_forward), PLZ_CALL(hard_forward_smallm), PLZ_CALL(hard_forward_bias), PLZ_CALL(eval_linear), PLZ_CALL(backward_dx),
                          PLZ_CALL(backward_dw_hard), PLZ_CALL(col_sum), PLZ_CALL(select_indices), PLZ_CALL(backward_dw_soft), {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_plz_torch", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__plz_torch(void) { return PyModule_Create(&kModule); }
