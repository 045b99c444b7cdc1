// Host side of an eager packed-Linear call, in C++: what a module's forward does per call is an output allocation, the
// current stream, a workspace look-up and one launch.  In Python that took 13 - 17 us, longer than the kernels.
//
// Three things live here: `Linear`, the prepared launches of one module (one per row count, up to 16 rows), `functional`,
// the prepared-problem cache of the decode_int*_linear functions, and `settled`, the record of weights that launches have
// already waited for.  The C ABI (include/qgemv_b200.h) does the work; nothing here knows about kernels.
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/ATen.h>
#include <ATen/autocast_mode.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/core/impl/LocalDispatchKeySet.h>

#include <algorithm>
#include <iterator>
#include <memory>
#include <mutex>
#include <optional>
#include <unordered_map>
#include <vector>

#include "../../include/qgemv_b200.h"

namespace {

using Opt = std::optional<at::Tensor>;

PyObject* g_workspace_fn = nullptr;                   // ops.ensure_workspace: (device index) -> tensor for the current stream
std::mutex g_mutex;
std::unordered_map<uint64_t, void*> g_workspace;      // (device, stream) -> workspace; the buffers live as long as the process

struct PyError {};                                    // a Python exception is set

PyObject* g_error_class = nullptr;                    // _cabi.QgemvError(code, message)

void check(int rc) {
    if (rc == QGEMV_OK) return;
    PyObject* e = PyObject_CallFunction(g_error_class, "is", rc, qgemv_error_string());
    if (e) { PyErr_SetObject(g_error_class, e); Py_DECREF(e); }
    throw PyError{};
}

// Called with the GIL held.
void* workspace(int device, cudaStream_t stream, size_t* bytes) {
    *bytes = qgemv_workspace_bytes(4, QGEMV_MAX_M, 1, 256, 128, 64);
    const uint64_t key = (reinterpret_cast<uint64_t>(stream) << 6) ^ (uint64_t)device;
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        auto it = g_workspace.find(key);
        if (it != g_workspace.end()) return it->second;
    }
    PyObject* t = PyObject_CallFunction(g_workspace_fn, "i", device);
    if (!t) throw PyError{};
    void* p = THPVariable_Unpack(t).data_ptr();
    Py_DECREF(t);
    std::lock_guard<std::mutex> lock(g_mutex);
    g_workspace[key] = p;
    return p;
}

Opt optional_tensor(PyObject* o) {
    if (!o || o == Py_None) return std::nullopt;
    return THPVariable_Unpack(o);
}

void fill(qgemv_problem& p, int bits, int64_t k_original, int group, int act, int kernel, const at::Tensor& packed, const at::Tensor& scales,
          const Opt& bias, const Opt& oidx, const Opt& ow, const Opt& ru, const Opt& rv) {
    p = qgemv_problem{};
    p.bits = bits; p.n = (int)packed.size(0); p.k_padded = (int)(packed.size(1) * (8 / bits)); p.k_original = (int)k_original;
    p.group = group; p.act = act; p.kernel = kernel & 0xff; p.debug = kernel >> 8;
    p.packed = packed.data_ptr<uint8_t>(); p.ldp = packed.stride(0);
    p.scales = scales.data_ptr(); p.lds = scales.stride(0);
    if (bias) p.bias = bias->data_ptr();
    if (oidx && oidx->numel()) {
        p.outliers = (int)oidx->numel();
        p.outlier_idx = oidx->data_ptr<int32_t>(); p.outlier_w = ow->data_ptr(); p.ldow = ow->stride(0);
    }
    if (ru && ru->numel()) {
        p.rank = (int)ru->size(1);
        p.res_u = ru->data_ptr(); p.ldu = ru->stride(0); p.res_v = rv->data_ptr(); p.ldv = rv->stride(0);
    }
}

// ---- settled weights ------------------------------------------------------------------------------------

// A launch may read weights before the preceding kernel of its stream has finished, unless that kernel may be what writes them.
// Weights are settled once a launch that waited for everything before it has seen them: from then on the version counter that
// their views share changes with every write that goes through the framework (a write through `.data` or a raw pointer leaves no
// trace on the host).  Inference tensors have no counter and are never settled.
// While a graph is captured nothing runs: what is recorded settles weights for launches recorded later (when the graph runs, all
// that was issued before it has finished), not for eager ones.
uint64_t g_failures = 0;                              // launches that were to wait and were not issued: nothing is settled any more
struct Settled {
    uint64_t version = ~0ull, failures = 0;
    bool eager = false;
    // Whether a launch has waited for this version; one has from now on (the caller's, which waits if this says no).
    template <typename Capturing> bool pass(uint64_t now, Capturing capturing) {
        const bool same = version == now && failures == g_failures;
        if (same && eager) return true;
        const bool cap = capturing(), was = same && cap;
        version = now;
        failures = g_failures;
        eager = !cap;
        return was;
    }
};
bool capturing_now() { return c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None; }      // current device's current stream

// By storage.  The weak reference keeps the address of a freed storage from being given to another one, so a match of addresses
// is the same storage.
struct Seen {
    c10::weak_intrusive_ptr<c10::StorageImpl> storage{c10::intrusive_ptr<c10::StorageImpl>()};
    Settled state;
};
std::unordered_map<const void*, Seen> g_seen;         // guarded by the GIL
constexpr size_t kMaxSeen = 8192;
size_t g_seen_sweep = 256;                            // entries of freed storages are dropped when this many are held

bool settle(const at::Tensor& t) {
    if (t.is_inference()) return false;
    const c10::Storage& storage = t.storage();
    const void* key = storage.unsafeGetStorageImpl();
    auto it = g_seen.find(key);
    if (it != g_seen.end()) return it->second.state.pass(t._version(), capturing_now);
    if (g_seen.size() >= g_seen_sweep) {
        for (auto i = g_seen.begin(); i != g_seen.end();) i = i->second.storage.expired() ? g_seen.erase(i) : std::next(i);
        if (g_seen.size() >= kMaxSeen) g_seen.clear();
        g_seen_sweep = std::min(kMaxSeen, std::max<size_t>(256, 2 * g_seen.size()));
    }
    return g_seen.emplace(key, Seen{storage.getWeakStorageImpl(), {}}).first->second.state.pass(t._version(), capturing_now);
}

// settled(tensor or None, ...): whether launches have waited for all of them; they count as settled from this call on
PyObject* settled(PyObject*, PyObject* const* a, Py_ssize_t n) {
    bool all = true;
    c10::cuda::OptionalCUDAGuard guard;
    try {
        for (Py_ssize_t i = 0; i < n; ++i) {
            if (a[i] == Py_None) continue;
            if (!THPVariable_Check(a[i])) { PyErr_SetString(PyExc_TypeError, "settled takes tensors"); return nullptr; }
            const at::Tensor& t = THPVariable_Unpack(a[i]);
            if (t.is_cuda() && c10::cuda::current_device() != t.get_device()) guard.set_index(t.get_device());
            all = settle(t) && all;
        }
    } catch (const std::exception& e) { PyErr_SetString(PyExc_RuntimeError, e.what()); return nullptr; }
    return PyBool_FromLong(all);
}

// forget(): a launch that was to wait was not issued
PyObject* forget(PyObject*, PyObject*) { ++g_failures; Py_RETURN_NONE; }
void check_launched(int rc) {
    if (rc != QGEMV_OK) ++g_failures;
    check(rc);
}

// ---- Linear ---------------------------------------------------------------------------------------------

enum Operand { kPacked, kScales, kBias, kOutlierIdx, kOutlierW, kResU, kResV, kOperands };

struct Linear {
    Opt operand[kOperands];                           // kept alive
    const void* address[kOperands] = {};              // where they were when `base` was filled
    bool valid = false;                               // `base` is filled: types, strides, shapes and devices are the kernels'
    bool counted = true;                              // all of them have version counters
    Settled settled;                                  // by the sum of the counters
    qgemv_problem base;
    int bits, group, act, kernel, device = -1;
    int64_t k_original, in_features, out_features, max_rows;
    struct Slot { std::vector<char> blob; bool usable = false; };
    std::unordered_map<int, Slot> slots;              // rows * 2 + bf16
};

// The kernels read raw memory: a module whose buffers were cast (`module.to(torch.bfloat16)`), or that was put together from
// something else, must not get here.  Its calls take the general route, which says what is wrong.
bool fits(const Linear& l) {
    const Opt* o = l.operand;
    auto matrix = [&](const Opt& t, at::ScalarType type, int64_t rows, int64_t cols) {
        return t && t->dim() == 2 && t->scalar_type() == type && t->is_cuda() && t->get_device() == o[kPacked]->get_device() && t->size(0) == rows &&
               t->size(1) >= cols && (t->size(1) == 1 || t->stride(1) == 1);
    };
    auto vector = [&](const Opt& t, at::ScalarType type, int64_t n) {
        return t && t->dim() == 1 && t->scalar_type() == type && t->is_cuda() && t->get_device() == o[kPacked]->get_device() && t->size(0) == n && (n < 2 || t->stride(0) == 1);
    };
    if (!o[kPacked] || !o[kPacked]->is_cuda() || o[kPacked]->dim() != 2 || l.group < 1) return false;
    const int64_t n = o[kPacked]->size(0), kpad = o[kPacked]->size(1) * (8 / l.bits);
    if (!matrix(o[kPacked], at::kByte, n, 1) || !matrix(o[kScales], at::kHalf, n, (kpad + l.group - 1) / l.group)) return false;
    if (o[kBias] && !vector(o[kBias], at::kHalf, n)) return false;
    if (o[kOutlierIdx]) {
        const int64_t oc = o[kOutlierIdx]->numel();
        if (!vector(o[kOutlierIdx], at::kInt, oc) || !matrix(o[kOutlierW], at::kHalf, n, oc)) return false;
    }
    if (o[kResU] || o[kResV])
        return o[kResU] && o[kResV] && o[kResU]->dim() == 2 && matrix(o[kResU], at::kHalf, n, 1) && matrix(o[kResV], at::kHalf, o[kResU]->size(1), l.k_original);
    return true;
}

// Fills `base` from the operands as they are now; what was prepared from earlier addresses goes.
void bind(Linear& l) {
    l.slots.clear();
    l.settled = {};
    l.counted = true;
    for (int i = 0; i < kOperands; ++i) {
        l.address[i] = l.operand[i] ? l.operand[i]->const_data_ptr() : nullptr;
        l.counted = l.counted && !(l.operand[i] && l.operand[i]->is_inference());
    }
    l.valid = fits(l);
    if (!l.valid) return;
    l.device = l.operand[kPacked]->get_device();
    fill(l.base, l.bits, l.k_original, l.group, l.act, l.kernel, *l.operand[kPacked], *l.operand[kScales], l.operand[kBias], l.operand[kOutlierIdx], l.operand[kOutlierW],
         l.operand[kResU], l.operand[kResV]);
}

// Whether `base` may be used; operands that were given other memory (`module.scales.data = ...`) are taken up.
bool bound(Linear& l) {
    for (int i = 0; i < kOperands; ++i)
        if (l.operand[i] && l.operand[i]->const_data_ptr() != l.address[i]) { bind(l); break; }
    return l.valid;
}

bool settle(Linear& l) {
    if (!l.counted) return false;
    uint64_t v = 0;
    for (const Opt& t : l.operand) if (t) v += t->_version();
    return l.settled.pass(v, capturing_now);
}

struct LinearObject { PyObject_HEAD Linear* self; };

void linear_dealloc(LinearObject* o) { delete o->self; Py_TYPE(o)->tp_free(reinterpret_cast<PyObject*>(o)); }

// Linear(bits, k_original, group, act, kernel, in_features, out_features, max_rows, packed, scales, bias, oidx, ow, ru, rv)
PyObject* linear_new(PyTypeObject* type, PyObject* args, PyObject*) {
    int bits, group, act, kernel;
    long long korig, in, out, max_rows;
    PyObject *packed, *scales, *bias, *oidx, *ow, *ru, *rv;
    if (!PyArg_ParseTuple(args, "iLiiiLLLOOOOOOO", &bits, &korig, &group, &act, &kernel, &in, &out, &max_rows, &packed, &scales, &bias, &oidx, &ow, &ru, &rv))
        return nullptr;
    if (bits != 2 && bits != 4) { PyErr_SetString(PyExc_ValueError, "bits must be 2 or 4"); return nullptr; }
    auto l = std::make_unique<Linear>();
    l->bits = bits; l->k_original = korig; l->group = group; l->act = act; l->kernel = kernel;
    try {
        PyObject* const given[kOperands] = {packed, scales, bias, oidx, ow, ru, rv};
        for (int i = 0; i < kOperands; ++i) l->operand[i] = optional_tensor(given[i]);
        bind(*l);
    } catch (const std::exception& e) { PyErr_SetString(PyExc_RuntimeError, e.what()); return nullptr; }
    l->in_features = in; l->out_features = out; l->max_rows = max_rows;
    auto* o = reinterpret_cast<LinearObject*>(type->tp_alloc(type, 0));
    if (o) o->self = l.release();
    return reinterpret_cast<PyObject*>(o);
}

// Whether something other than the plain forward pass wants to see the operators of this call: a transform (vmap, jvp, grad), a
// tracer, a dispatch mode, a batched or functional wrapper of x.
bool observed(const at::Tensor& x) {
    constexpr c10::DispatchKeySet watching({c10::DispatchKey::Python, c10::DispatchKey::PythonTLSSnapshot, c10::DispatchKey::PythonDispatcher, c10::DispatchKey::Functionalize,
                                            c10::DispatchKey::Tracer, c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::FuncTorchVmapMode,
                                            c10::DispatchKey::FuncTorchDynamicLayerFrontMode, c10::DispatchKey::FuncTorchDynamicLayerBackMode});
    return !((x.key_set() | c10::impl::tls_local_dispatch_key_set().included_) & watching).empty();
}

// Beyond the rows of the fused GEMV a module is an expression of differentiable operators; the fused GEMM stands for it only where
// nobody asks for derivatives, or through autocast for other types (the residual's products are fp16 ones).
bool plain_forward(const Linear& l, const at::Tensor& x) {
    if ((at::GradMode::is_enabled() && x.requires_grad()) || x._fw_grad(/*level=*/0).defined()) return false;
    return !at::autocast::is_autocast_enabled(at::kCUDA) ||
           (at::autocast::get_autocast_dtype(at::kCUDA) == x.scalar_type() && (x.scalar_type() == at::kHalf || !l.operand[kResU]));
}

// The fused GEMM makes a tile's weights once for every 256 rows of x, the expression once, and multiplies at the library's rate:
// many rows over long K are the expression's again.  Eager calls, GEMM against expression: 2048 rows x 14336 columns (N = 4096) 276
// against 293 us, 4096 x 4096 (N = 14336) 677 against 763; 4096 x 8192 (N = 28672) 2117 against 1986, 8192 x 4096 1462 against 1404.
bool many(int64_t rows, int64_t k) { return rows * k > (int64_t(30) << 20); }

// call(x): the result, or None where the caller has to take its general route (shape, type, device, layout; operands that are
// not the kernels').
PyObject* linear_call(LinearObject* o, PyObject* arg) {
    Linear& l = *o->self;
    if (!THPVariable_CheckExact(arg)) Py_RETURN_NONE;
    try {
        const at::Tensor& x = THPVariable_Unpack(arg);
        if (observed(x) || !bound(l)) Py_RETURN_NONE;
        const int64_t dims = x.dim();
        const auto dtype = x.scalar_type();
        if (dims < 1 || !x.is_cuda() || x.get_device() != l.device || x.size(-1) != l.in_features || !x.is_contiguous() ||
            (dtype != at::kHalf && dtype != at::kBFloat16))
            Py_RETURN_NONE;
        const int64_t rows = x.numel() / l.in_features;
        const bool batch = rows > l.max_rows;
        if (batch && !plain_forward(l, x)) Py_RETURN_NONE;
        if (rows < 1 || rows > (1 << 24) || (!batch && reinterpret_cast<uintptr_t>(x.data_ptr()) % 16)) Py_RETURN_NONE;
        c10::cuda::OptionalCUDAGuard guard;
        if (c10::cuda::current_device() != l.device) guard.set_index(l.device);
        const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(l.device).stream();
        size_t ws_bytes = 0;
        void* ws = workspace(l.device, stream, &ws_bytes);
        const bool bf16 = dtype == at::kBFloat16;
        auto result = [&]() {
            if (dims == 2) return at::empty({rows, l.out_features}, x.options());
            std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end());
            shape.back() = l.out_features;
            return at::empty(shape, x.options());
        };
        if (batch) {                                  // weights are read after the layout kernel, which starts in stream order
            qgemv_problem p = l.base;
            if ((p.kernel & 0xff) == QGEMV_KERNEL_SIMT || many(rows, l.k_original)) Py_RETURN_NONE;
            p.m = (int)rows; p.x_dtype = bf16 ? QGEMV_BF16 : QGEMV_F16;
            p.x = x.data_ptr(); p.ldx = l.in_features;
            p.y = x.data_ptr(); p.ldy = l.out_features;
            p.workspace = ws; p.workspace_bytes = ws_bytes;
            const size_t bytes = qgemv_batch_scratch_bytes(&p);
            if (!bytes) Py_RETURN_NONE;
            at::Tensor y = result(), scratch = at::empty({(int64_t)bytes}, x.options().dtype(at::kByte));
            p.y = y.data_ptr();
            check(qgemv_run_batch(&p, scratch.data_ptr(), bytes, stream));
            return THPVariable_Wrap(std::move(y));
        }
        Linear::Slot& slot = l.slots[(int)rows * 2 + bf16];
        if (slot.blob.empty()) {
            slot.blob.resize(qgemv_prepared_bytes());
            qgemv_problem p = l.base;
            p.m = (int)rows; p.x_dtype = bf16 ? QGEMV_BF16 : QGEMV_F16;
            p.x = x.data_ptr(); p.ldx = l.in_features;
            p.y = x.data_ptr(); p.ldy = l.out_features;       // a valid address for the plan; the launch names the real one
            p.workspace = ws; p.workspace_bytes = ws_bytes;
            const int rc = qgemv_prepare(&p, slot.blob.data());
            slot.usable = rc == QGEMV_OK;
            if (rc != QGEMV_OK && rc != QGEMV_ERR_ALIGN) check(rc);
        }
        if (!slot.usable) Py_RETURN_NONE;
        at::Tensor y = result();
        check_launched(qgemv_launch_prepared(slot.blob.data(), x.data_ptr(), y.data_ptr(), ws, !settle(l), stream));
        return THPVariable_Wrap(std::move(y));
    } catch (const PyError&) { return nullptr; }
    catch (const std::exception& e) { PyErr_SetString(PyExc_RuntimeError, e.what()); return nullptr; }
}

PyObject* linear_tp_call(PyObject* self, PyObject* args, PyObject* kw) {
    if (PyTuple_GET_SIZE(args) != 1 || (kw && PyDict_GET_SIZE(kw))) { PyErr_SetString(PyExc_TypeError, "one activation tensor expected"); return nullptr; }
    return linear_call(reinterpret_cast<LinearObject*>(self), PyTuple_GET_ITEM(args, 0));
}

// settled(): as the function of this name, for the module's operands (a launch made without this object)
PyObject* linear_settled(LinearObject* o, PyObject*) {
    Linear& l = *o->self;
    try {
        c10::cuda::OptionalCUDAGuard guard;
        if (!bound(l)) Py_RETURN_FALSE;
        if (c10::cuda::current_device() != l.device) guard.set_index(l.device);
        return PyBool_FromLong(settle(l));
    } catch (const std::exception& e) { PyErr_SetString(PyExc_RuntimeError, e.what()); return nullptr; }
}

PyMethodDef linear_methods[] = {{"settled", reinterpret_cast<PyCFunction>(linear_settled), METH_NOARGS, "whether launches have waited for the operands as they are"},
                                {"call", reinterpret_cast<PyCFunction>(linear_call), METH_O, "call(x) -> y, or None for the caller's general route"}, {nullptr, nullptr, 0, nullptr}};
PyTypeObject LinearType = {PyVarObject_HEAD_INIT(nullptr, 0)};

// ---- functional -----------------------------------------------------------------------------------------

// A problem is reused when addresses AND shapes of the operands of this call are the ones it was built from; the cache
// holds no tensor alive.  Whether the operands are settled is asked apart from that: by their storages and versions.
struct Key {
    uint64_t w[20];
    bool operator==(const Key& o) const { return std::equal(w, w + 20, o.w); }
};
struct KeyHash {
    size_t operator()(const Key& k) const {
        uint64_t h = 1469598103934665603ull;
        for (uint64_t v : k.w) { h ^= v + 0x9e3779b97f4a7c15ull + (h << 6) + (h >> 2); }
        return (size_t)h;
    }
};
constexpr size_t kMaxProblems = 256;
struct Problem {
    qgemv_problem p;
    Seen seen[7];                                     // packed, scales, bias, oidx, ow, ru, rv
    bool settle(PyObject* const* a) {
        bool all = true;
        for (int i = 0; i < 7; ++i) {
            if (a[6 + i] == Py_None) continue;
            const at::Tensor& t = THPVariable_Unpack(a[6 + i]);
            if (t.is_inference()) { all = false; continue; }
            const c10::Storage& storage = t.storage();
            if (seen[i].storage._unsafe_get_target() != storage.unsafeGetStorageImpl()) seen[i] = Seen{storage.getWeakStorageImpl(), {}};
            all = seen[i].state.pass(t._version(), capturing_now) && all;
        }
        return all;
    }
};
std::unordered_map<Key, Problem, KeyHash> g_problems;      // guarded by the GIL

// functional(bits, group, k_original, act, kernel, x, packed, scales, bias, oidx, ow, ru, rv) -> y, or None for the general route
PyObject* functional(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 13) { PyErr_SetString(PyExc_TypeError, "functional takes 13 arguments"); return nullptr; }
    long v[5];
    for (int i = 0; i < 5; ++i) { v[i] = PyLong_AsLong(a[i]); if (v[i] == -1 && PyErr_Occurred()) return nullptr; }
    for (int i = 5; i < 13; ++i) {
        if (a[i] == Py_None && i > 7) continue;
        if (!THPVariable_CheckExact(a[i])) Py_RETURN_NONE;
    }
    try {
        const at::Tensor &x = THPVariable_Unpack(a[5]), &packed = THPVariable_Unpack(a[6]), &scales = THPVariable_Unpack(a[7]);
        const auto dtype = x.scalar_type();
        const int cpb = 8 / (int)v[0];
        if (!x.is_cuda() || x.dim() != 2 || x.size(0) < 1 || x.size(0) > QGEMV_MAX_M || x.stride(1) != 1 || (dtype != at::kHalf && dtype != at::kBFloat16) ||
            packed.dim() != 2 || packed.scalar_type() != at::kByte || packed.stride(1) != 1 || packed.size(1) * cpb != x.size(1) ||
            scales.dim() != 2 || scales.scalar_type() != at::kHalf || scales.stride(1) != 1)
            Py_RETURN_NONE;
        const int dev = x.get_device();
        Key key{};
        uint64_t* w = key.w;
        *w++ = (uint64_t)v[0] | (uint64_t)v[1] << 8 | (uint64_t)v[3] << 40 | (uint64_t)dev << 48 | (uint64_t)(dtype == at::kHalf) << 56;
        *w++ = (uint64_t)v[2] | (uint64_t)v[4] << 32;
        *w++ = (uint64_t)x.size(0) | (uint64_t)x.stride(0) << 8;
        *w++ = (uint64_t)packed.data_ptr(); *w++ = (uint64_t)packed.size(0) | (uint64_t)packed.size(1) << 32; *w++ = packed.stride(0);
        *w++ = (uint64_t)scales.data_ptr(); *w++ = scales.stride(0);
        for (int i = 8; i < 13; ++i) {
            if (a[i] == Py_None) { *w++ = 0; *w++ = 0; continue; }
            const at::Tensor& t = THPVariable_Unpack(a[i]);
            if (!t.is_cuda() || t.get_device() != dev || t.scalar_type() != (i == 9 ? at::kInt : at::kHalf) || (t.dim() && t.numel() && t.stride(-1) != 1)) Py_RETURN_NONE;
            *w++ = (uint64_t)t.data_ptr();
            *w++ = t.dim() == 2 ? (uint64_t)t.size(0) << 40 ^ (uint64_t)t.size(1) << 20 ^ (uint64_t)t.stride(0) : (uint64_t)t.numel();
        }
        auto it = g_problems.find(key);
        if (it == g_problems.end()) {
            if (packed.get_device() != dev || scales.get_device() != dev || scales.size(0) != packed.size(0) || scales.size(1) * v[1] != x.size(1)) Py_RETURN_NONE;
            Problem entry;
            qgemv_problem& p = entry.p;
            const Opt oi = optional_tensor(a[9]), ow = optional_tensor(a[10]), ru = optional_tensor(a[11]), rv = optional_tensor(a[12]);
            if ((oi && oi->numel() && (!ow || ow->dim() != 2)) || (ru && ru->numel() && (ru->dim() != 2 || !rv || rv->dim() != 2))) Py_RETURN_NONE;
            fill(p, (int)v[0], v[2], (int)v[1], (int)v[3], (int)v[4], packed, scales, optional_tensor(a[8]), oi, ow, ru, rv);
            p.m = (int)x.size(0); p.x_dtype = dtype == at::kHalf ? QGEMV_F16 : QGEMV_BF16;
            p.ldx = x.stride(0); p.ldy = p.n;
            if (g_problems.size() >= kMaxProblems) g_problems.clear();
            it = g_problems.emplace(key, std::move(entry)).first;
        }
        qgemv_problem& p = it->second.p;
        c10::cuda::OptionalCUDAGuard guard;
        if (c10::cuda::current_device() != dev) guard.set_index(dev);
        const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev).stream();
        size_t ws_bytes = 0;
        void* ws = workspace(dev, stream, &ws_bytes);
        at::Tensor y = at::empty({x.size(0), p.n}, x.options());
        p.x = x.data_ptr(); p.y = y.data_ptr(); p.workspace = ws; p.workspace_bytes = ws_bytes;
        check_launched((it->second.settle(a) ? qgemv_run : qgemv_run_ordered)(&p, stream));
        return THPVariable_Wrap(std::move(y));
    } catch (const PyError&) { return nullptr; }
    catch (const std::exception& e) { PyErr_SetString(PyExc_RuntimeError, e.what()); return nullptr; }
}

// ---- quantiser ------------------------------------------------------------------------------------------

// pack(weight, bits, group, rms, first, last, steps) -> (packed, scales), or None where the caller has to prepare the operands (or raise)
PyObject* pack(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 7) { PyErr_SetString(PyExc_TypeError, "pack takes 7 arguments"); return nullptr; }
    const long bits = PyLong_AsLong(a[1]), group = PyLong_AsLong(a[2]), steps = PyLong_AsLong(a[6]);
    const double first = PyFloat_AsDouble(a[4]), last = PyFloat_AsDouble(a[5]);
    if (PyErr_Occurred()) return nullptr;
    if (!THPVariable_CheckExact(a[0]) || (a[3] != Py_None && !THPVariable_CheckExact(a[3]))) Py_RETURN_NONE;
    try {
        const at::Tensor& w = THPVariable_Unpack(a[0]);
        const auto type = w.scalar_type();
        if (observed(w) || !w.is_cuda() || w.dim() != 2 || w.numel() == 0 || w.stride(1) != 1 || w.stride(0) < w.size(1) || w.size(0) > 0x7fffffff || w.size(1) > 0x7fffffff ||
            (type != at::kHalf && type != at::kBFloat16 && type != at::kFloat) || steps < 1 || steps > QGEMV_PACK_MAX_SPACED || group < 1)
            Py_RETURN_NONE;
        const float* rms = nullptr;
        if (a[3] != Py_None) {
            const at::Tensor& r = THPVariable_Unpack(a[3]);
            if (observed(r) || !r.is_cuda() || r.get_device() != w.get_device() || r.scalar_type() != at::kFloat || r.dim() != 1 || (r.numel() > 1 && r.stride(0) != 1) ||
                r.numel() < w.size(1))
                Py_RETURN_NONE;
            rms = static_cast<const float*>(r.data_ptr());
        }
        c10::cuda::OptionalCUDAGuard guard;
        if (c10::cuda::current_device() != w.get_device()) guard.set_index(w.get_device());
        const int64_t rows = w.size(0), k = w.size(1), ng = (k + group - 1) / group;
        at::Tensor packed = at::empty({rows, ng * group * bits / 8}, w.options().dtype(at::kByte)), scales = at::empty({rows, ng}, w.options().dtype(at::kHalf));
        check(qgemv_pack_spaced((int)bits, w.data_ptr(), w.stride(0), type == at::kHalf ? QGEMV_F16 : type == at::kBFloat16 ? QGEMV_BF16 : QGEMV_F32, (int)rows, (int)k, (int)group,
                                rms, (float)first, (float)last, (int)steps, static_cast<uint8_t*>(packed.data_ptr()), scales.data_ptr(),
                                c10::cuda::getCurrentCUDAStream(w.get_device()).stream()));
        PyObject* const pp = THPVariable_Wrap(std::move(packed));
        PyObject* const ps = THPVariable_Wrap(std::move(scales));
        return Py_BuildValue("(NN)", pp, ps);
    } catch (const PyError&) { return nullptr; }
    catch (const std::exception& e) { PyErr_SetString(PyExc_RuntimeError, e.what()); return nullptr; }
}

// setup(ensure_workspace, error_class)
PyObject* setup(PyObject*, PyObject* args) {
    PyObject *fn, *err;
    if (!PyArg_ParseTuple(args, "OO", &fn, &err)) return nullptr;
    Py_INCREF(fn); Py_INCREF(err);
    g_workspace_fn = fn; g_error_class = err;
    Py_RETURN_NONE;
}

PyMethodDef module_methods[] = {
    {"setup", setup, METH_VARARGS, "setup(ensure_workspace, error_class)"},
    {"forget", forget, METH_NOARGS, "no weights are settled any more"},
    {"settled", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(settled)), METH_FASTCALL, "whether launches have waited for these weights"},
    {"functional", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(functional)), METH_FASTCALL, "prepared-problem call of the decode_int*_linear functions"},
    {"pack", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(pack)), METH_FASTCALL, "quantiser call for operands as the kernel takes them"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_native", "Host side of eager packed-Linear calls", -1, module_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) {
    LinearType.tp_name = "ai_accel_studio_b200._native.Linear";
    LinearType.tp_basicsize = sizeof(LinearObject);
    LinearType.tp_dealloc = reinterpret_cast<destructor>(linear_dealloc);
    LinearType.tp_flags = Py_TPFLAGS_DEFAULT;
    LinearType.tp_new = linear_new;
    LinearType.tp_call = linear_tp_call;
    LinearType.tp_methods = linear_methods;
    LinearType.tp_doc = "Prepared launches of one packed Linear module, one per row count";
    if (PyType_Ready(&LinearType) < 0) return nullptr;
    PyObject* m = PyModule_Create(&module_def);
    if (!m) return nullptr;
    Py_INCREF(&LinearType);
    PyModule_AddObject(m, "Linear", reinterpret_cast<PyObject*>(&LinearType));
    return m;
}
