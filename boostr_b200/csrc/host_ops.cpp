// Python entry points of the quantized operators, as a CPython extension (boostr_b200/_hostops.so).
//
// A decode-sized product keeps the GPU busy for 2-15 us, and the Python form of a call (argument checks on torch tensors,
// ctypes conversions, device and stream context managers, the scratch look-up) took 12-16 us of host time, so eager calls
// were bound by it: Q4_0 4096 x 4096 at M = 1 ran at 16.1 us a call around a 4.9 us kernel.  Here a call is one
// METH_FASTCALL function: it reads the tensors' fields, allocates the output from torch's caching allocator, takes the
// scratch buffer of (device, stream) and enters the C ABI (include/b200q.h); nothing is kept from one call for the next.
//
// Only well-formed calls are served: anything unusual (a tensor subclass, a non-contiguous or misaligned activation, a
// shape or type the operators reject) returns NotImplemented and the Python form of the operator takes the call, which
// also raises the error texts.  A non-zero status of the C ABI is returned as an int and raised by the caller.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/version.h>

#include <algorithm>
#include <map>
#include <memory>
#include <mutex>
#include <optional>
#include <utility>
#include <vector>

#include "../../include/b200q.h"

namespace {

// What the C ABI needs of a QuantTensor; held by its Python object as a capsule.
struct WeightRef {
    at::Tensor storage;
    int format = 0;
    bool matrix = false;   // a 2-D [n, k] weight
    size_t n = 0, k = 0;
    std::vector<int64_t> shape;
    size_t numel = 0;
};
constexpr const char* CAPSULE = "boostr_b200.WeightRef";
PyObject* s_ref = nullptr;  // interned "_ref"

WeightRef* ref_of_capsule(PyObject* o) {
    if (!PyCapsule_CheckExact(o)) return nullptr;
    return static_cast<WeightRef*>(PyCapsule_GetPointer(o, CAPSULE));
}
// The WeightRef of a QuantTensor, held with its capsule until the end of the call (the attribute is made by the first call
// that asks for it, on any thread); none (and no Python error) when the object has none.
class Ref {
    PyObject* capsule_;
    WeightRef* w_ = nullptr;

  public:
    explicit Ref(PyObject* qt) : capsule_(PyObject_GetAttr(qt, s_ref)) {
        if (capsule_) w_ = ref_of_capsule(capsule_);
        if (!w_) PyErr_Clear();
    }
    Ref(const Ref&) = delete;
    ~Ref() { Py_XDECREF(capsule_); }
    explicit operator bool() const { return w_ != nullptr; }
    WeightRef* operator->() const { return w_; }
};

// The objects of a list or tuple at the time of the call, held until its end: reading an attribute of one of them runs Python,
// and other threads run during the launches, so the list itself may change meanwhile.
struct Items {
    static constexpr Py_ssize_t MAX = 16;
    PyObject* o[MAX];
    Py_ssize_t n = 0;
    Items() = default;
    Items(const Items&) = delete;
    ~Items() {
        for (Py_ssize_t i = 0; i < n; ++i) Py_DECREF(o[i]);
    }
    bool take(PyObject* seq) {
        if (!PyList_CheckExact(seq) && !PyTuple_CheckExact(seq)) return false;
        if (PySequence_Fast_GET_SIZE(seq) > MAX) return false;
        for (; n < PySequence_Fast_GET_SIZE(seq); ++n) o[n] = Py_NewRef(PySequence_Fast_GET_ITEM(seq, n));
        return true;
    }
};

// Scratch buffers of eager calls: one per (device, stream), grown on demand.  Calls on one stream run in order, so they may
// share a buffer; the entry's mutex keeps the launches of two threads on one stream from interleaving inside a call, and
// the call's own reference keeps a buffer that another thread replaces alive until its launches are enqueued.
// A call that is being captured into a graph takes none of them: a replay runs whenever and on whichever stream its owner
// launches it, beside eager calls and other graphs, and its addresses outlive the growth of a shared buffer.  Its
// scratch is allocated for the call, from the memory pool of the graph, which keeps it.
struct Scratch {
    std::mutex m;
    at::Tensor buf;
};
std::mutex g_scratch_mutex;
// never destroyed: its tensors must not outlive the CUDA context at exit
auto& g_scratch = *new std::map<std::pair<int, cudaStream_t>, std::unique_ptr<Scratch>>;
Scratch& scratch_of(int device, cudaStream_t st) {
    std::lock_guard<std::mutex> g(g_scratch_mutex);
    auto& e = g_scratch[{device, st}];
    if (!e) e = std::make_unique<Scratch>();
    return *e;
}

at::Tensor empty(c10::IntArrayRef shape, at::ScalarType t, c10::Device dev) {
    return at::Tensor(at::detail::empty_cuda(shape, t, dev, std::nullopt));
}

int dtype_code(at::ScalarType t) {
    switch (t) {
    case at::kFloat: return B200Q_F32;
    case at::kBFloat16: return B200Q_BF16;
    case at::kHalf: return B200Q_F16;
    case at::kDouble: return B200Q_F64;
    default: return -1;
    }
}
at::ScalarType scalar_type(long code) {
    return code == B200Q_F32 ? at::kFloat : code == B200Q_BF16 ? at::kBFloat16 : code == B200Q_F16 ? at::kHalf : at::kDouble;
}

// A contiguous, 16-byte aligned F32 / BF16 CUDA activation [..., k]; false: not one.
struct Act {
    const at::Tensor* t = nullptr;
    size_t m = 0, k = 0;
    int dt = 0;
    c10::Device dev{c10::DeviceType::CUDA, 0};
};
bool act_of(PyObject* o, Act& a) {
    if (!THPVariable_CheckExact(o)) return false;
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || t.dim() < 1 || !t.is_contiguous()) return false;
    a.dt = dtype_code(t.scalar_type());
    if (a.dt != B200Q_F32 && a.dt != B200Q_BF16) return false;
    a.k = (size_t)t.size(-1);
    if (a.k == 0 || t.numel() == 0 || (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15)) return false;
    a.m = (size_t)t.numel() / a.k;
    a.t = &t;
    a.dev = t.device();
    return true;
}
bool weight_fits(const Ref& w, const Act& a) { return w && w->matrix && w->k == a.k && w->storage.device() == a.dev; }

// The output: `given` (validated) or a new tensor [..., n]; false: `given` does not fit.
bool out_of(PyObject* given, const Act& a, size_t n, at::ScalarType t, at::Tensor& out) {
    const auto sz = a.t->sizes();
    if (given == Py_None) {
        c10::SmallVector<int64_t, 6> shape(sz.begin(), sz.end());
        shape.back() = (int64_t)n;
        out = empty(shape, t, a.dev);
        return true;
    }
    if (!THPVariable_CheckExact(given)) return false;
    out = THPVariable_Unpack(given);
    if (!out.is_cuda() || out.device() != a.dev || out.scalar_type() != t || !out.is_contiguous() || out.dim() != a.t->dim() ||
        out.size(-1) != (int64_t)n)
        return false;
    for (int64_t i = 0; i + 1 < out.dim(); ++i)
        if (out.size(i) != sz[i]) return false;
    return true;
}

// Makes `dev` current for the scope when it is not (a no-op in a one-GPU process).
struct DeviceScope {
    std::optional<c10::cuda::CUDAGuard> guard;
    explicit DeviceScope(c10::Device d) {
        if (c10::cuda::current_device() != d.index()) guard.emplace(d);
    }
};

bool capturing(cudaStream_t st) {
    cudaStreamCaptureStatus s = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &s) == cudaSuccess) return s != cudaStreamCaptureStatusNone;
    cudaGetLastError();  // the legacy stream beside another thread's capture: the launch itself will say so
    return false;
}

// Other Python threads run while this lives.
struct NoGil {
    PyThreadState* state = PyEval_SaveThread();
    NoGil() = default;
    NoGil(const NoGil&) = delete;
    ~NoGil() { PyEval_RestoreThread(state); }
};

// Runs call(scratch pointer, scratch bytes, stream) without the GIL, with at least `need` bytes of scratch.
template <typename F>
int with_scratch(c10::Device dev, size_t need, F&& call) {
    const cudaStream_t st = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    if (!need) {
        NoGil nogil;
        return call(static_cast<void*>(nullptr), (size_t)0, st);
    }
    if (capturing(st)) {
        const at::Tensor buf = empty({(int64_t)need}, at::kByte, dev);
        NoGil nogil;
        return call(buf.data_ptr(), need, st);
    }
    Scratch& s = scratch_of(dev.index(), st);
    NoGil nogil;
    std::lock_guard<std::mutex> g(s.m);
    if (!s.buf.defined() || (size_t)s.buf.numel() < need) {
        s.buf = at::Tensor();  // back to the allocator first: a grown buffer may reuse its memory
        s.buf = empty({(int64_t)std::max<size_t>(need, (size_t)1 << 20)}, at::kByte, dev);
    }
    return call(s.buf.data_ptr(), (size_t)s.buf.numel(), st);
}

PyObject* not_served() { Py_RETURN_NOTIMPLEMENTED; }
PyObject* result(int rc, const at::Tensor& out) {
    if (rc != B200Q_OK) return PyLong_FromLong(rc);
    return THPVariable_Wrap(out);
}
template <typename F>
PyObject* guarded(F&& f) {  // no C++ exception may cross into the interpreter
    try {
        return f();
    } catch (...) {
        PyErr_Clear();
        return not_served();  // the Python form runs the same call and raises what torch raises
    }
}

// make_ref(storage, format id, shape) -> capsule
PyObject* make_ref(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 3 || !THPVariable_Check(args[0]) || !PyTuple_Check(args[2])) {
        PyErr_SetString(PyExc_TypeError, "make_ref(storage, format, shape)");
        return nullptr;
    }
    auto r = std::make_unique<WeightRef>();
    r->storage = THPVariable_Unpack(args[0]);
    r->format = (int)PyLong_AsLong(args[1]);
    r->numel = 1;
    for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(args[2]); ++i) {
        r->shape.push_back((int64_t)PyLong_AsLongLong(PyTuple_GET_ITEM(args[2], i)));
        r->numel *= (size_t)r->shape.back();
    }
    if (PyErr_Occurred()) return nullptr;
    if (r->shape.size() == 2 && r->storage.is_cuda()) {
        r->matrix = true;
        r->n = (size_t)r->shape[0];
        r->k = (size_t)r->shape[1];
    }
    return PyCapsule_New(r.release(), CAPSULE, [](PyObject* c) { delete static_cast<WeightRef*>(PyCapsule_GetPointer(c, CAPSULE)); });
}

// quant_matmul(act, weight, out dtype code, out or None)
PyObject* quant_matmul(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        Act a;
        if (nargs != 4 || !act_of(args[0], a)) return not_served();
        const Ref w(args[1]);
        if (!weight_fits(w, a)) return not_served();
        const long odt = PyLong_AsLong(args[2]);
        DeviceScope dev(a.dev);
        at::Tensor out;
        if (!out_of(args[3], a, w->n, scalar_type(odt), out)) return not_served();
        const size_t need = b200q_workspace_bytes(B200Q_OP_QUANT_MATMUL, w->format, a.m, a.k, w->n);
        const int rc = with_scratch(a.dev, need, [&](void* ws, size_t bytes, cudaStream_t st) {
            return b200q_quant_matmul(w->format, a.t->data_ptr(), a.dt, w->storage.data_ptr(), out.data_ptr(), (int)odt, a.m, a.k, w->n, ws,
                                      bytes, st);
        });
        return result(rc, out);
    });
}

// quant_matmul_batch(act, norm weight or None, eps, weights, out dtype code, outs or None) -> list
PyObject* quant_matmul_batch(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        Act a;
        if (nargs != 6 || !act_of(args[0], a)) return not_served();
        Items weights, given;
        if (!weights.take(args[3]) || weights.n < 1 || (args[5] != Py_None && (!given.take(args[5]) || given.n != weights.n))) return not_served();
        const Py_ssize_t nw = weights.n;
        const long odt = PyLong_AsLong(args[4]);
        DeviceScope dev(a.dev);
        int fmts[Items::MAX];
        const void* wp[Items::MAX];
        size_t ns[Items::MAX];
        void* op[Items::MAX];
        at::Tensor outs[Items::MAX];
        size_t need = 0;
        for (Py_ssize_t i = 0; i < nw; ++i) {
            const Ref w(weights.o[i]);
            if (!weight_fits(w, a)) return not_served();
            fmts[i] = w->format;
            wp[i] = w->storage.data_ptr();
            ns[i] = w->n;
            need = std::max(need, b200q_workspace_bytes(B200Q_OP_QUANT_MATMUL, w->format, a.m, a.k, w->n));
        }
        const float* norm = nullptr;
        float eps = 0.f;
        if (args[1] != Py_None) {
            if (!THPVariable_CheckExact(args[1])) return not_served();
            const at::Tensor& t = THPVariable_Unpack(args[1]);
            if (!t.is_cuda() || t.device() != a.dev || t.scalar_type() != at::kFloat || (size_t)t.numel() != a.k || !t.is_contiguous()) return not_served();
            norm = t.data_ptr<float>();
            eps = (float)PyFloat_AsDouble(args[2]);
            need += (a.m * a.k * 4 + 255) / 256 * 256;
        }
        if (PyErr_Occurred()) {
            PyErr_Clear();
            return not_served();
        }
        for (Py_ssize_t i = 0; i < nw; ++i) {
            if (!out_of(given.n ? given.o[i] : Py_None, a, ns[i], scalar_type(odt), outs[i])) return not_served();
            op[i] = outs[i].data_ptr();
        }
        const int rc = with_scratch(a.dev, need, [&](void* ws, size_t bytes, cudaStream_t st) {
            if (norm)
                return b200q_rmsnorm_quant_matmul_batch((int)nw, fmts, wp, ns, op, a.t->data_ptr(), norm, eps, a.dt, (int)odt, a.m, a.k, ws, bytes, st);
            return b200q_quant_matmul_batch((int)nw, fmts, wp, ns, op, a.t->data_ptr(), a.dt, (int)odt, a.m, a.k, ws, bytes, st);
        });
        if (rc != B200Q_OK) return PyLong_FromLong(rc);
        PyObject* list = PyList_New(nw);
        if (!list) return nullptr;
        for (Py_ssize_t i = 0; i < nw; ++i) {
            PyObject* o = THPVariable_Wrap(outs[i]);  // the given tensor itself, or the new one where None was given
            if (!o) {
                Py_DECREF(list);
                return nullptr;
            }
            PyList_SET_ITEM(list, i, o);
        }
        return list;
    });
}

// quant_swiglu(act, gate, up, out dtype code, out or None)
PyObject* quant_swiglu(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        Act a;
        if (nargs != 5 || !act_of(args[0], a)) return not_served();
        const Ref g(args[1]), u(args[2]);
        if (!weight_fits(g, a) || !weight_fits(u, a) || g->format != u->format || g->n != u->n) return not_served();
        const long odt = PyLong_AsLong(args[3]);
        DeviceScope dev(a.dev);
        at::Tensor out;
        if (!out_of(args[4], a, g->n, scalar_type(odt), out)) return not_served();
        const size_t need = b200q_workspace_bytes(B200Q_OP_QUANT_SWIGLU, g->format, a.m, a.k, g->n);
        const int rc = with_scratch(a.dev, need, [&](void* ws, size_t bytes, cudaStream_t st) {
            return b200q_quant_swiglu(g->format, a.t->data_ptr(), a.dt, g->storage.data_ptr(), u->storage.data_ptr(), out.data_ptr(), (int)odt, a.m,
                                      a.k, g->n, ws, bytes, st);
        });
        return result(rc, out);
    });
}

// quant_mlp(act, gate, up, down, out dtype code, out or None)
PyObject* quant_mlp(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        Act a;
        if (nargs != 6 || !act_of(args[0], a)) return not_served();
        const Ref g(args[1]), u(args[2]), d(args[3]);
        if (!weight_fits(g, a) || !weight_fits(u, a) || g->format != u->format || g->n != u->n || !d || !d->matrix || d->k != g->n ||
            d->storage.device() != a.dev)
            return not_served();
        const long odt = PyLong_AsLong(args[4]);
        DeviceScope dev(a.dev);
        at::Tensor out;
        if (!out_of(args[5], a, d->n, scalar_type(odt), out)) return not_served();
        const size_t need = b200q_mlp_workspace_bytes(g->format, d->format, a.m, a.k, g->n, d->n);
        const int rc = with_scratch(a.dev, need, [&](void* ws, size_t bytes, cudaStream_t st) {
            return b200q_quant_mlp(g->format, g->storage.data_ptr(), u->storage.data_ptr(), d->format, d->storage.data_ptr(), a.t->data_ptr(), a.dt,
                                   out.data_ptr(), (int)odt, a.m, a.k, g->n, d->n, ws, bytes, st);
        });
        return result(rc, out);
    });
}

// dequantize(weight, out dtype code)
PyObject* dequantize(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        if (nargs != 2) return not_served();
        const Ref w(args[0]);
        const size_t block = w ? b200q_block_size(w->format) : 0;
        if (!block || !w->storage.is_cuda()) return not_served();  // 0: not a format of this library
        const long odt = PyLong_AsLong(args[1]);
        const c10::Device d = w->storage.device();
        DeviceScope dev(d);
        at::Tensor out = empty(w->shape, scalar_type(odt), d);
        const size_t nblocks = w->numel / block;
        const int rc = with_scratch(d, 0, [&](void*, size_t, cudaStream_t st) {
            return b200q_dequantize(w->format, w->storage.data_ptr(), nblocks, out.data_ptr(), (int)odt, st);
        });
        return result(rc, out);
    });
}

PyMethodDef methods[] = {
    {"make_ref", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(make_ref)), METH_FASTCALL, nullptr},
    {"quant_matmul", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(quant_matmul)), METH_FASTCALL, nullptr},
    {"quant_matmul_batch", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(quant_matmul_batch)), METH_FASTCALL, nullptr},
    {"quant_swiglu", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(quant_swiglu)), METH_FASTCALL, nullptr},
    {"quant_mlp", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(quant_mlp)), METH_FASTCALL, nullptr},
    {"dequantize", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(dequantize)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_hostops", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__hostops(void) {
    s_ref = PyUnicode_InternFromString("_ref");
    PyObject* m = PyModule_Create(&module);
    if (m && PyModule_AddStringConstant(m, "torch_version", TORCH_VERSION) != 0) Py_CLEAR(m);
    return m;
}
