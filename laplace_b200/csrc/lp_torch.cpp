// lp_torch.cpp - the host side of the device-pointer calls for programs that hold their data in torch tensors.
//
// A decode step is a handful of kernels of 3 to 10 us. The checks, the allocation of the results, the look-up of the stream
// and the ctypes call of device.py took 13 us a call, so that the GPU waited for the host (layer of one row: 43 us of
// kernels in 68 us). Here the same steps are a few native calls.
//
// Every function returns the result, or None for anything but a plain, valid call that succeeded: device.py then takes its
// general path, which checks the arguments, repeats the call and raises. Nothing is kept from one call for the next.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "laplace_cuda.h"

namespace {

struct Entries {
    decltype(&laplace_cuda_gemm_dev) gemm;
    decltype(&laplace_cuda_gemm_multi_dev) gemm_multi;
    decltype(&laplace_cuda_moe_gemv_dev) moe_gemv;
    decltype(&laplace_cuda_lm_head_dev) lm_head;
    decltype(&laplace_cuda_moe_route_dev) moe_route;
    decltype(&laplace_cuda_moe_ffn_dev) moe_ffn;
} g;
int g_device = -1;

// GGUF blocks: values and bytes; 0: a type that the general path sorts out
void block_of(long type, long& elems, long& bytes) {
    switch (type) {
        case 0: elems = 1; bytes = 4; break;             // F32
        case 1: case 30: elems = 1; bytes = 2; break;    // F16, BF16
        case 2: elems = 32; bytes = 18; break;           // Q4_0
        case 6: elems = 32; bytes = 22; break;           // Q5_0
        case 8: elems = 32; bytes = 34; break;           // Q8_0
        case 10: elems = 256; bytes = 84; break;         // Q2_K
        case 11: elems = 256; bytes = 110; break;        // Q3_K
        case 12: elems = 256; bytes = 144; break;        // Q4_K
        case 13: elems = 256; bytes = 176; break;        // Q5_K
        case 14: elems = 256; bytes = 210; break;        // Q6_K
        default: elems = 0; bytes = 0;
    }
}
bool whole_rows(const at::Tensor& w, long type, long K, long N) {
    long elems, bytes;
    block_of(type, elems, bytes);
    return elems && K > 0 && N > 0 && K % elems == 0 && w.numel() >= N * (K / elems) * bytes;
}

bool tensor(PyObject* o, at::ScalarType type, const at::Tensor*& t) {
    if (!THPVariable_CheckExact(o)) return false;        // subclasses go the general way
    t = &THPVariable_Unpack(o);
    return t->is_cuda() && t->scalar_type() == type && t->is_contiguous() && t->get_device() == g_device;
}
bool number(PyObject* o, long& v) {
    v = PyLong_AsLong(o);
    if (v == -1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
    return v >= 0 && v < (1L << 31);
}
bool real(PyObject* o, double& v) {
    v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) { PyErr_Clear(); return false; }
    return true;
}
bool ready() { return g_device >= 0 && c10::cuda::current_device() == g_device; }
// torch's default stream has handle 0, which the library reads as "its own stream": it is passed as cudaStreamLegacy
void* stream() {
    cudaStream_t s = c10::cuda::getCurrentCUDAStream().stream();
    return s ? static_cast<void*>(s) : reinterpret_cast<void*>(1);
}
at::Tensor fresh(at::IntArrayRef sizes, at::ScalarType type) { return at::empty(sizes, at::TensorOptions().dtype(type).device(at::kCUDA, g_device)); }

template <class F>
PyObject* guarded(F&& f) {
    try {
        return f();
    } catch (...) {        // an allocation that failed, a tensor without storage: the general path meets it again and raises
        PyErr_Clear();
        Py_RETURN_NONE;
    }
}
// Runs f without the interpreter lock, which is back however f ends. Only the library's own call belongs in f: data_ptr() throws
// for a tensor without storage (inside torch.vmap, torch.func.grad and the like), so pointers are taken before.
struct Unlocked {
    PyThreadState* st = PyEval_SaveThread();
    Unlocked() = default;
    Unlocked(const Unlocked&) = delete;
    Unlocked& operator=(const Unlocked&) = delete;
    ~Unlocked() { PyEval_RestoreThread(st); }
};
template <class F>
int unlocked(F&& f) {
    Unlocked lock;
    return f();
}
template <class T> T* ptr(const at::Tensor& t) { return static_cast<T*>(t.data_ptr()); }

// gemm(x, w, type, M, K, N, y or None)
PyObject* py_gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        const at::Tensor *x, *w, *y = nullptr;
        long type, M, K, N;
        if (n != 7 || !ready() || !tensor(a[0], at::kFloat, x) || !tensor(a[1], at::kByte, w) || !number(a[2], type) || !number(a[3], M) ||
            !number(a[4], K) || !number(a[5], N) || (a[6] != Py_None && !tensor(a[6], at::kFloat, y)) || x->numel() < M * K || !whole_rows(*w, type, K, N) ||
            (y && y->numel() < M * N))
            Py_RETURN_NONE;
        const at::Tensor out = y ? *y : fresh({M, N}, at::kFloat);
        const auto* px = ptr<const float>(*x);
        const auto* pw = ptr<const uint8_t>(*w);
        auto* po = ptr<float>(out);
        void* st = stream();
        if (unlocked([&] { return g.gemm(px, pw, type, po, M, K, N, st); }))
            Py_RETURN_NONE;
        if (y) { Py_INCREF(a[6]); return a[6]; }
        return THPVariable_Wrap(out);
    });
}

// gemm_multi(x, ws, type, M, K, Ns, norm_weight or None, eps)
PyObject* py_gemm_multi(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        const at::Tensor *x, *norm = nullptr, *w;
        long type, M, K;
        double eps;
        if (n != 8 || !ready() || !tensor(a[0], at::kFloat, x) || !PyList_CheckExact(a[1]) || !(PyList_CheckExact(a[5]) || PyTuple_CheckExact(a[5])) || !number(a[2], type) ||
            !number(a[3], M) || !number(a[4], K) || (a[6] != Py_None && !tensor(a[6], at::kFloat, norm)) || !real(a[7], eps) || x->numel() < M * K || (norm && norm->numel() < K))
            Py_RETURN_NONE;
        const Py_ssize_t count = PyList_GET_SIZE(a[1]);
        if (count < 1 || count > 8 || PySequence_Fast_GET_SIZE(a[5]) != count) Py_RETURN_NONE;
        laplace_cuda_matrix mats[8];
        at::Tensor ys[8];
        for (Py_ssize_t i = 0; i < count; ++i) {
            long N;
            if (!tensor(PyList_GET_ITEM(a[1], i), at::kByte, w) || !number(PySequence_Fast_GET_ITEM(a[5], i), N) || !whole_rows(*w, type, K, N)) Py_RETURN_NONE;
            ys[i] = fresh({M, N}, at::kFloat);
            mats[i] = laplace_cuda_matrix{ptr<const uint8_t>(*w), ptr<float>(ys[i]), static_cast<int>(N)};
        }
        const auto* px = ptr<const float>(*x), *pn = norm ? ptr<const float>(*norm) : nullptr;
        void* st = stream();
        if (unlocked([&] { return g.gemm_multi(px, pn, static_cast<float>(eps), nullptr, mats, static_cast<int>(count), type, M, K, st); }))
            Py_RETURN_NONE;
        PyObject* list = PyList_New(count);
        if (!list) return nullptr;
        for (Py_ssize_t i = 0; i < count; ++i) {
            PyObject* o = THPVariable_Wrap(ys[i]);
            if (!o) { Py_DECREF(list); return nullptr; }
            PyList_SET_ITEM(list, i, o);
        }
        return list;
    });
}

// moe_gemv(x, w, type, expert_idx, K, N, per_expert_x, y or None)
PyObject* py_moe_gemv(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        const at::Tensor *x, *w, *idx, *y = nullptr;
        long type, K, N;
        if (n != 8 || !ready() || !tensor(a[0], at::kFloat, x) || !tensor(a[1], at::kByte, w) || !number(a[2], type) || !tensor(a[3], at::kInt, idx) || !number(a[4], K) ||
            !number(a[5], N) || (a[7] != Py_None && !tensor(a[7], at::kFloat, y)))
            Py_RETURN_NONE;
        const int per = PyObject_IsTrue(a[6]);
        if (per < 0) { PyErr_Clear(); Py_RETURN_NONE; }
        const long e = idx->numel();
        if (x->numel() < (per ? e : 1) * K || (y && y->numel() < e * N)) Py_RETURN_NONE;
        const at::Tensor out = y ? *y : fresh({e, N}, at::kFloat);
        const auto* px = ptr<const float>(*x);
        const auto* pw = ptr<const uint8_t>(*w);
        const auto* pi = ptr<const int>(*idx);
        auto* po = ptr<float>(out);
        void* st = stream();
        if (unlocked([&] { return g.moe_gemv(px, pw, type, pi, e, po, K, N, per, st); }))
            Py_RETURN_NONE;
        if (y) { Py_INCREF(a[7]); return a[7]; }
        return THPVariable_Wrap(out);
    });
}

// lm_head(x, w, type, M, K, N, softcap)
PyObject* py_lm_head(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        const at::Tensor *x, *w;
        long type, M, K, N;
        double cap;
        if (n != 7 || !ready() || !tensor(a[0], at::kFloat, x) || !tensor(a[1], at::kByte, w) || !number(a[2], type) || !number(a[3], M) || !number(a[4], K) ||
            !number(a[5], N) || !real(a[6], cap) || x->numel() < M * K || !whole_rows(*w, type, K, N))
            Py_RETURN_NONE;
        const at::Tensor out = fresh({M, N}, at::kFloat);
        const auto* px = ptr<const float>(*x);
        const auto* pw = ptr<const uint8_t>(*w);
        auto* po = ptr<float>(out);
        void* st = stream();
        if (unlocked([&] { return g.lm_head(px, pw, type, po, M, K, N, static_cast<float>(cap), st); }))
            Py_RETURN_NONE;
        return THPVariable_Wrap(out);
    });
}

// moe_route(logits, top_k)
PyObject* py_moe_route(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        const at::Tensor* l;
        long k;
        if (n != 2 || !ready() || !tensor(a[0], at::kFloat, l) || l->dim() != 2 || !number(a[1], k)) Py_RETURN_NONE;
        const at::Tensor idx = fresh({l->size(0), k}, at::kInt), wts = fresh({l->size(0), k}, at::kFloat);
        const auto* pl = ptr<const float>(*l);
        const long T = l->size(0), E = l->size(1);
        auto* pi = ptr<int>(idx);
        auto* pw = ptr<float>(wts);
        void* st = stream();
        if (unlocked([&] { return g.moe_route(pl, T, E, k, pi, pw, st); }))
            Py_RETURN_NONE;
        return Py_BuildValue("NN", THPVariable_Wrap(idx), THPVariable_Wrap(wts));
    });
}

// moe_ffn(x, w_gate_up, w_down, type_gate_up, type_down, top_idx, top_w, experts, hidden, inter, activation)
PyObject* py_moe_ffn(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        const at::Tensor *x, *wg, *wd, *idx, *tw;
        long tg, td, E, H, I, act;
        if (n != 11 || !ready() || !tensor(a[0], at::kFloat, x) || !tensor(a[1], at::kByte, wg) || !tensor(a[2], at::kByte, wd) || !number(a[3], tg) || !number(a[4], td) ||
            !tensor(a[5], at::kInt, idx) || !tensor(a[6], at::kFloat, tw) || !number(a[7], E) || !number(a[8], H) || !number(a[9], I) || !number(a[10], act) ||
            idx->dim() != 2 || tw->sizes() != idx->sizes() || x->dim() != 2 || x->size(0) != idx->size(0) || x->size(1) != H)
            Py_RETURN_NONE;
        const long T = idx->size(0), k = idx->size(1);
        const at::Tensor out = fresh({T, H}, at::kFloat);
        const auto* px = ptr<const float>(*x), *pt = ptr<const float>(*tw);
        const auto* pg = ptr<const uint8_t>(*wg), *pd = ptr<const uint8_t>(*wd);
        const auto* pi = ptr<const int>(*idx);
        auto* po = ptr<float>(out);
        void* st = stream();
        if (unlocked([&] { return g.moe_ffn(px, pg, pd, tg, td, pi, pt, nullptr, T, k, E, H, I, act, po, nullptr, st); }))
            Py_RETURN_NONE;
        return THPVariable_Wrap(out);
    });
}

// bind(device, addresses of the six entry points in the order of Entries)
PyObject* py_bind(PyObject*, PyObject* args) {
    int dev;
    unsigned long long p[6];
    if (!PyArg_ParseTuple(args, "iKKKKKK", &dev, &p[0], &p[1], &p[2], &p[3], &p[4], &p[5])) return nullptr;
    g.gemm = reinterpret_cast<decltype(g.gemm)>(p[0]);
    g.gemm_multi = reinterpret_cast<decltype(g.gemm_multi)>(p[1]);
    g.moe_gemv = reinterpret_cast<decltype(g.moe_gemv)>(p[2]);
    g.lm_head = reinterpret_cast<decltype(g.lm_head)>(p[3]);
    g.moe_route = reinterpret_cast<decltype(g.moe_route)>(p[4]);
    g.moe_ffn = reinterpret_cast<decltype(g.moe_ffn)>(p[5]);
    g_device = dev;
    Py_RETURN_NONE;
}

#define LP_FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_##name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {LP_FAST(gemm), LP_FAST(gemm_multi), LP_FAST(moe_gemv), LP_FAST(lm_head), LP_FAST(moe_route), LP_FAST(moe_ffn),
                         {"bind", py_bind, METH_VARARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&module); }
