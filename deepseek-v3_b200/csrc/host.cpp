// Native host path of the Python operators: argument checks, output allocation and the call into libdsv3_b200.so in
// one CPython call each.
//
// Why it exists: a decode-sized operator runs for 2-8 us on a B200, while the same call through ctypes (device guard,
// stream lookup, three or four framework calls for the outputs, pointer conversions) kept the host busy for 14-20 us,
// so every small call was bound by its own launch.  Here a call costs the two allocations and the launch itself.
// The extension adds nothing to the C ABI: it fills in the same arguments a C host would.
//
// Threads and streams: every entry point is called with the GIL held and releases it only around the library call;
// the split-K workspaces are keyed on (device, stream, capture), and calls that share one are ordered by their stream.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/DefaultDtype.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <array>
#include <exception>
#include <memory>
#include <algorithm>
#include <vector>

#include "dsv3_b200.h"

namespace {

PyObject* g_error_class = nullptr;   // dsv3_b200.Dsv3Error

PyObject* g_oom_class = nullptr;     // torch.OutOfMemoryError

// A Python exception is already set.
struct PythonError {};

[[noreturn]] void raise(PyObject* type, const char* msg) {
    PyErr_SetString(type, msg);
    throw PythonError{};
}

void require(bool cond, const char* assertion) {
    if (!cond) raise(PyExc_AssertionError, assertion);
}

void check(int status) {
    if (status == DSV3_OK) return;
    PyObject* msg = PyUnicode_FromFormat("%s (%d): %s", dsv3_strerror(status), status, dsv3_last_error());
    if (msg) {
        PyObject* exc = PyObject_CallFunction(g_error_class, "iO", status, msg);
        Py_DECREF(msg);
        if (exc) {
            PyErr_SetObject(g_error_class, exc);
            Py_DECREF(exc);
        }
    }
    throw PythonError{};
}

const at::Tensor& tensor_arg(PyObject* o) {
    if (!THPVariable_Check(o)) raise(PyExc_TypeError, "expected a torch.Tensor");
    return THPVariable_Unpack(o);
}

int scale_fmt_arg(PyObject* o) {
    return (PyUnicode_Check(o) && PyUnicode_CompareWithASCIIString(o, "ue8m0") == 0) ? DSV3_SCALE_FMT_UE8M0
                                                                                     : DSV3_SCALE_FMT_FP32;
}

// All tensors of a call live on one CUDA device; returns it.
template <typename... Ts>
c10::Device require_cuda(const at::Tensor& first, const Ts&... rest) {
    const c10::Device dev = first.device();
    const at::Tensor* all[] = {&first, &rest...};
    for (const at::Tensor* t : all) {
        if (!t->is_cuda()) {
            PyErr_Format(PyExc_RuntimeError, "dsv3_b200 runs on CUDA tensors only (there is no CPU path); got a %s tensor",
                         c10::DeviceTypeName(t->device().type(), true).c_str());
            throw PythonError{};
        }
        if (t->device() != dev) raise(PyExc_RuntimeError, "all tensors of one call must be on the same device");
    }
    return dev;
}

void require_bf16_default() {
    const auto dt = c10::get_default_dtype_as_scalartype();
    if (dt != at::kBFloat16) {
        PyErr_Format(PyExc_NotImplementedError,
                     "the CUDA path writes bfloat16 only; call torch.set_default_dtype(torch.bfloat16) as every entry point of "
                     "the reference does (default dtype is %s)", c10::toString(dt));
        throw PythonError{};
    }
}

at::Tensor new_cuda(at::IntArrayRef sizes, at::ScalarType dt, c10::Device dev) {
    return at::detail::empty_cuda(sizes, dt, dev, std::nullopt);
}

// `like`'s sizes with the last one replaced.
at::Tensor new_cuda_last(const at::Tensor& like, int64_t last, at::ScalarType dt) {
    c10::SmallVector<int64_t, 6> sizes(like.sizes().begin(), like.sizes().end());
    if (sizes.empty()) sizes.push_back(last); else sizes.back() = last;
    return new_cuda(sizes, dt, like.device());
}

int64_t last_dim(const at::Tensor& t) {
    if (t.dim() == 0) raise(PyExc_IndexError, "Dimension specified as -1 but tensor has no dimensions");
    return t.sizes().back();
}

PyObject* wrap(at::Tensor t) { return THPVariable_Wrap(std::move(t)); }

PyObject* wrap_pair(at::Tensor a, at::Tensor b) {
    PyObject* first = wrap(std::move(a));
    PyObject* second = first ? wrap(std::move(b)) : nullptr;
    PyObject* tup = second ? PyTuple_New(2) : nullptr;
    if (!tup) {
        Py_XDECREF(first);
        Py_XDECREF(second);
        return nullptr;
    }
    PyTuple_SET_ITEM(tup, 0, first);
    PyTuple_SET_ITEM(tup, 1, second);
    return tup;
}

// Runs a library call with the tensors' device current and without the GIL; raises what it reports.
template <typename F>
void call_library(c10::Device dev, F&& f) {
    c10::cuda::OptionalCUDAGuard guard;
    if (dev.index() != c10::cuda::current_device()) guard.set_device(dev);
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    int status;
    {
        PyThreadState* save = PyEval_SaveThread();
        status = f(static_cast<dsv3_stream_t>(stream));
        PyEval_RestoreThread(save);
    }
    check(status);
}

// Which capture a stream takes part in: 0 for none, otherwise a number that no other capture of the process has.
unsigned long long capture_of(cudaStream_t stream) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    unsigned long long id = 0;
    if (cudaStreamGetCaptureInfo(stream, &status, &id) != cudaSuccess) {
        (void)cudaGetLastError();          // the legacy stream next to a capture: not capturing itself
        return 0;
    }
    return status == cudaStreamCaptureStatusNone ? 0 : id + 1;
}

// ------------------------------------------------------------------ split-K workspaces, one per (device, stream, capture)
struct Workspace {
    int device;
    cudaStream_t stream;
    unsigned long long capture;      // 0: eager calls
    at::Tensor mem;
};
// Ordered by last use; beyond kKeptWorkspaces the one used longest ago goes back to torch's allocator, which hands its
// memory out again in the order of the stream it was used on.
// A graph has a workspace of its own: its header is cleared by a node of that graph, which nothing else may rely on (the
// graph may be replayed late, never, or after another one), and a replay may run beside eager calls on the stream the graph
// was captured on.  Its memory comes from the graph's pool, which stays reserved as long as the graph lives, so the
// reference is given up when the stream is next seen in another capture or in none.
// (never destroyed: at process exit the CUDA context may already be gone)
std::vector<Workspace>& g_workspaces = *new std::vector<Workspace>;
constexpr size_t kKeptWorkspaces = 16;

// The header of a workspace must be zero on first use; every call leaves it zero again.  The caller holds the returned tensor
// until its launches have been issued: while it has released the GIL for them, another thread may replace or drop the
// entry, and only memory given up after the launches is handed out behind them in the stream's order.
at::Tensor workspace(c10::Device dev, size_t bytes) {
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    const unsigned long long capture = capture_of(stream);
    const auto here = [&](const Workspace& w) { return w.device == dev.index() && w.stream == stream; };
    g_workspaces.erase(std::remove_if(g_workspaces.begin(), g_workspaces.end(),
                                      [&](const Workspace& w) { return here(w) && w.capture != 0 && w.capture != capture; }),
                       g_workspaces.end());
    auto it = std::find_if(g_workspaces.begin(), g_workspaces.end(), [&](const Workspace& w) { return here(w) && w.capture == capture; });
    const bool found = it != g_workspaces.end();
    if (!found || static_cast<size_t>(it->mem.numel()) < bytes) {
        // (a graph's: small enough for torch to place it beside the graph's other tensors; a device allocation of its own, and
        // giving it back, cost 0.8 ms per capture)
        int64_t size = std::max<int64_t>(static_cast<int64_t>(bytes), (capture ? 8ll : 16ll) << 20);
        if (found) size = std::max<int64_t>(size, 2 * it->mem.numel());
        c10::cuda::OptionalCUDAGuard guard(dev);
        at::Tensor mem = new_cuda({size}, at::kByte, dev);
        if (cudaMemsetAsync(mem.data_ptr(), 0, DSV3_WORKSPACE_HEADER_BYTES, stream) != cudaSuccess)
            raise(PyExc_RuntimeError, "could not clear the header of a new split-K workspace");
        if (found) {
            it->mem = std::move(mem);
        } else {
            if (g_workspaces.size() >= kKeptWorkspaces) g_workspaces.erase(g_workspaces.begin());
            g_workspaces.push_back({dev.index(), stream, capture, std::move(mem)});
            it = g_workspaces.end() - 1;
        }
    }
    if (it + 1 != g_workspaces.end()) std::rotate(it, it + 1, g_workspaces.end());
    return g_workspaces.back().mem;
}

// ------------------------------------------------------------------ operators
std::pair<at::Tensor, at::Tensor> quantise(const at::Tensor& x, int64_t block, int fmt) {
    require(x.is_contiguous(), "Input tensor must be contiguous");
    const int64_t K = last_dim(x);
    if (block <= 0 || K % block != 0) {
        PyErr_Format(PyExc_AssertionError, "Last dimension size must be divisible by block_size (block_size=%lld)",
                     static_cast<long long>(block));
        throw PythonError{};
    }
    const c10::Device dev = require_cuda(x);
    if (x.scalar_type() != at::kBFloat16) {
        PyErr_Format(PyExc_NotImplementedError, "act_quant takes bfloat16 activations (got %s)", c10::toString(x.scalar_type()));
        throw PythonError{};
    }
    at::Tensor y = new_cuda(x.sizes(), at::kFloat8_e4m3fn, dev);
    at::Tensor s = new_cuda_last(x, K / block, at::kFloat);
    const int64_t rows = K ? x.numel() / K : 0;
    const void* xp = x.const_data_ptr();
    void* yp = y.data_ptr();
    float* sp = static_cast<float*>(s.data_ptr());
    call_library(dev, [&](dsv3_stream_t st) { return dsv3_act_quant(xp, rows, K, static_cast<int>(block), fmt, yp, sp, st); });
    return {std::move(y), std::move(s)};
}

at::Tensor gemm(const at::Tensor& a, const at::Tensor& a_s, const at::Tensor& b, const at::Tensor& b_s) {
    require(a.is_contiguous() && b.is_contiguous(), "Input tensors must be contiguous");
    require(a_s.is_contiguous() && b_s.is_contiguous(), "Scaling factor tensors must be contiguous");
    const c10::Device dev = require_cuda(a, a_s, b, b_s);
    if (a.element_size() != 1 || b.element_size() != 1 || a_s.scalar_type() != at::kFloat || b_s.scalar_type() != at::kFloat)
        raise(PyExc_NotImplementedError, "fp8_gemm takes 1-byte FP8 operands and float32 scales");
    const int64_t K = last_dim(a);
    if (K == 0) raise(PyExc_ZeroDivisionError, "integer division or modulo by zero");
    const int64_t M = a.numel() / K, N = b.size(0);
    require_bf16_default();
    at::Tensor c = new_cuda_last(a, N, at::kBFloat16);
    const size_t need = dsv3_fp8_gemm_workspace_bytes(M, N, K);
    const at::Tensor held = need ? workspace(dev, need) : at::Tensor();
    void* ws = need ? held.data_ptr() : nullptr;
    const size_t ws_bytes = need ? static_cast<size_t>(held.numel()) : 0;
    const void *ap = a.const_data_ptr(), *bp = b.const_data_ptr();
    const float *asp = static_cast<const float*>(a_s.const_data_ptr()), *bsp = static_cast<const float*>(b_s.const_data_ptr());
    void* cp = c.data_ptr();
    call_library(dev, [&](dsv3_stream_t st) { return dsv3_fp8_gemm(ap, asp, bp, bsp, M, N, K, cp, ws, ws_bytes, st); });
    return c;
}

at::Tensor linear_small(const at::Tensor& x, const at::Tensor& w, const at::Tensor& s, int fmt) {
    require(x.is_contiguous() && w.is_contiguous() && s.is_contiguous(), "Input tensors must be contiguous");
    const c10::Device dev = require_cuda(x, w, s);
    if (x.scalar_type() != at::kBFloat16 || w.element_size() != 1 || s.scalar_type() != at::kFloat)
        raise(PyExc_NotImplementedError, "fp8_linear takes bfloat16 activations, a 1-byte FP8 weight and float32 scales");
    const int64_t K = last_dim(x);
    const int64_t M = K ? x.numel() / K : 0, N = w.size(0);
    require_bf16_default();
    at::Tensor c = new_cuda_last(x, N, at::kBFloat16);
    const void *xp = x.const_data_ptr(), *wp = w.const_data_ptr();
    const float* sp = static_cast<const float*>(s.const_data_ptr());
    void* cp = c.data_ptr();
    call_library(dev, [&](dsv3_stream_t st) { return dsv3_fp8_linear(xp, M, K, wp, sp, N, fmt, cp, st); });
    return c;
}

// ------------------------------------------------------------------ the FP8 branch of linear()
// Quantisations of the two most recent activation tensors (see linear_seam.py for when an entry may be reused).
struct Remembered {
    c10::weak_intrusive_ptr<at::TensorImpl, c10::UndefinedTensorImpl> x;
    const void* data;
    c10::SmallVector<int64_t, 6> sizes;
    int64_t version;          // -1: a tensor without a modification counter
    int64_t block;
    int fmt;
    cudaStream_t stream;
    unsigned long long capture;   // a graph's quantisation is computed at its replays: for that capture only; and the other way round
    at::Tensor q, s;
};
std::vector<Remembered>& g_memo = *new std::vector<Remembered>;     // at most two, most recent first
PyObject* g_stats = nullptr;        // the seam's counters, a dict
PyObject *g_key_calls, *g_key_reused, *g_key_fused, *g_attr_scale;
PyObject *g_attr_dict, *g_key_forward, *g_key_hooks, *g_key_pre_hooks, *g_key_compiled;

void count(PyObject* key) {
    PyObject* old = g_stats ? PyDict_GetItemWithError(g_stats, key) : nullptr;
    if (!old) return;
    PyObject* now = PyLong_FromLong(PyLong_AsLong(old) + 1);
    if (!now || PyDict_SetItem(g_stats, key, now) != 0) PyErr_Clear();
    Py_XDECREF(now);
}

void remember(const at::Tensor& x, int64_t block, int fmt, bool assume_no_inplace, const at::Tensor& q, const at::Tensor& s) {
    const bool counted = !x.is_inference();
    if (!counted && !assume_no_inplace) return;
    if (g_memo.size() > 1) g_memo.pop_back();
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(x.device().index()).stream();
    g_memo.insert(g_memo.begin(),
                  Remembered{decltype(Remembered::x)(x.getIntrusivePtr()), x.const_data_ptr(), {x.sizes().begin(), x.sizes().end()},
                             counted ? static_cast<int64_t>(x._version()) : -1, block, fmt, stream, capture_of(stream), q, s});
}

std::pair<at::Tensor, at::Tensor> quantise_remembered(const at::Tensor& x, int64_t block, int fmt, bool assume_no_inplace) {
    const bool counted = !x.is_inference();
    if ((!counted && !assume_no_inplace) || !x.is_cuda()) {
        count(g_key_calls);
        return quantise(x, block, fmt);
    }
    const int64_t version = counted ? static_cast<int64_t>(x._version()) : -1;
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(x.device().index()).stream();
    for (size_t i = 0; i < g_memo.size(); ++i) {
        Remembered& e = g_memo[i];
        // a weak reference keeps the TensorImpl's address from being reused, so equal addresses mean the same tensor
        if (e.x._unsafe_get_target() == x.unsafeGetTensorImpl() && e.version == version && e.data == x.const_data_ptr() &&
            e.block == block && e.fmt == fmt && e.stream == stream && x.sizes() == at::IntArrayRef(e.sizes) && e.capture == capture_of(stream)) {
            count(g_key_reused);
            if (i) std::swap(g_memo[0], g_memo[i]);
            return {g_memo[0].q, g_memo[0].s};
        }
    }
    auto r = quantise(x, block, fmt);
    count(g_key_calls);
    remember(x, block, fmt, assume_no_inplace, r.first, r.second);
    return r;
}

// ------------------------------------------------------------------ an MLP whose Linears are plain
// w2(swiglu_quant(w1(x), w3(x))) in three launches: the quantisation of x, w1 and w3 with everything in front of w2, w2; or, with
// more tokens, in four: w1 and w3 in one launch, which fills the SMs' last round better than two.
// Undefined where the separate launches are faster: in a graph, where only the device counts, or from here, where the host's launches do too.
at::Tensor mlp(const at::Tensor& x, const at::Tensor (&w)[3], const at::Tensor (&s)[3], int x_fmt, int h_fmt, bool assume_no_inplace) {
    const int64_t K = last_dim(x), M = K ? x.numel() / K : 0, N = w[0].size(0);
    if (w[0].dim() != 2 || w[0].sizes() != w[1].sizes() || w[0].size(1) != K) return {};
    const bool fused = dsv3_swiglu_linear_pays(M, N, K) ||
                       (dsv3_swiglu_linear_saves_launches(M, N, K) && x.is_cuda() &&
                        capture_of(c10::cuda::getCurrentCUDAStream(x.device().index()).stream()) == 0);
    if (!fused && (N % 128 != 0 || !dsv3_fp8_gemm_two_pays(M, N, K))) return {};
    for (int i = 0; i < 2; ++i) {
        require(w[i].is_contiguous(), "Input tensors must be contiguous");
        require(s[i].is_contiguous(), "Scaling factor tensors must be contiguous");
        if (w[i].element_size() != 1 || s[i].scalar_type() != at::kFloat) raise(PyExc_NotImplementedError, "fp8_gemm takes 1-byte FP8 operands and float32 scales");
        if (reinterpret_cast<uintptr_t>(w[i].const_data_ptr()) % 16 != 0) return {};        // (the tcgen05 kernels' limit)
    }
    require_bf16_default();
    auto q = quantise_remembered(x, 128, x_fmt, assume_no_inplace);
    const c10::Device dev = require_cuda(q.first, w[0], s[0], w[1], s[1]);
    at::Tensor h, hs;
    const void *a = q.first.const_data_ptr(), *p1 = w[0].const_data_ptr(), *p3 = w[1].const_data_ptr();
    auto f32 = [](const at::Tensor& t) { return static_cast<const float*>(t.const_data_ptr()); };
    const float *as = f32(q.second), *s1 = f32(s[0]), *s3 = f32(s[1]);
    if (!fused) {
        // (what is no longer read is given back at once, as the separate launches give it back: w2's result may take its place)
        at::Tensor y1 = new_cuda_last(x, N, at::kBFloat16), y3 = new_cuda_last(x, N, at::kBFloat16);
        void *y1p = y1.data_ptr(), *y3p = y3.data_ptr();
        call_library(dev, [&](dsv3_stream_t st) { return dsv3_fp8_gemm_two(a, as, p1, s1, p3, s3, M, N, K, y1p, y3p, st); });
        q = {};
        h = new_cuda_last(x, N, at::kFloat8_e4m3fn);
        hs = new_cuda_last(x, N / 128, at::kFloat);
        void* hp = h.data_ptr();
        float* hsp = static_cast<float*>(hs.data_ptr());
        call_library(dev, [&](dsv3_stream_t st) { return dsv3_swiglu_quant(y1p, y3p, M, N, h_fmt, hp, hsp, st); });
        y1.reset();
        y3.reset();
        return gemm(h, hs, w[2], s[2]);
    }
    h = new_cuda_last(x, N, at::kFloat8_e4m3fn);
    hs = new_cuda_last(x, N / 128, at::kFloat);
    const size_t need = dsv3_swiglu_linear_workspace_bytes(M, N, K);
    const at::Tensor held = need ? workspace(dev, need) : at::Tensor();
    void* ws = need ? held.data_ptr() : nullptr;
    const size_t ws_bytes = need ? static_cast<size_t>(held.numel()) : 0;
    void* hp = h.data_ptr();
    float* hsp = static_cast<float*>(hs.data_ptr());
    call_library(dev, [&](dsv3_stream_t st) { return dsv3_swiglu_linear(a, as, p1, s1, p3, s3, M, N, K, h_fmt, hp, hsp, ws, ws_bytes, st); });
    return gemm(h, hs, w[2], s[2]);
}

// ------------------------------------------------------------------ expert layer
// Device tables of the local experts' projections and what they depend on.  The tables hold addresses, so before every
// pass the host must know that the experts are still the ones they were built from.  Looking every weight up through
// its module costs 0.3 us each (230 us for 256 experts); instead the dictionaries the look-ups went through are watched
// for changes, and only the storage addresses of the weights and scales are compared (`param.data = ...` changes no
// dictionary).  They are kept as Python objects: an object's tensor may be exchanged (torch.utils.swap_tensors).
uint64_t g_dict_changes = 1;         // bumped whenever a watched dictionary changes
int g_watcher = -1;

#if PY_VERSION_HEX >= 0x030C0000
int on_dict_change(PyDict_WatchEvent, PyObject*, PyObject*, PyObject*) {
    ++g_dict_changes;
    return 0;
}
#endif

struct LookUp {
    PyObject *dict, *key, *value;    // dict[key] is value (dict kept alive; value compared by identity)
};

struct Experts {
    int n, start, fmt;
    int64_t dim, inter;
    at::Tensor table1, table3, table2;
    PyObject* list;                  // the experts when they are a plain list, else null
    std::vector<PyObject*> members;  // its members [start, start + n)
    std::vector<LookUp> lookups;
    uint64_t seen = 0;               // g_dict_changes when the look-ups were last verified
    std::vector<std::pair<PyObject*, const void*>> tensors;     // weights and scales with the addresses in the tables
    ~Experts() {
        Py_XDECREF(list);
        for (auto& t : tensors) Py_DECREF(t.first);
        for (PyObject* m : members) Py_DECREF(m);
        for (LookUp& l : lookups) {
            Py_DECREF(l.dict);
            Py_DECREF(l.key);
            Py_DECREF(l.value);
        }
    }
    bool current() {
        if (list) {
            for (int i = 0; i < n; ++i)
                if (start + i >= PyList_GET_SIZE(list) || PyList_GET_ITEM(list, start + i) != members[i]) return false;
        }
        if (g_watcher < 0 || seen != g_dict_changes) {
            for (const LookUp& l : lookups)
                if (PyDict_GetItemWithError(l.dict, l.key) != l.value) return false;
            seen = g_dict_changes;
        }
        for (const auto& t : tensors)
            if (THPVariable_Unpack(t.first).const_data_ptr() != t.second) return false;
        return true;
    }
};

const char* kExpertsName = "dsv3_b200.experts";
void free_experts(PyObject* c) { delete static_cast<Experts*>(PyCapsule_GetPointer(c, kExpertsName)); }
Experts* experts_arg(PyObject* c) {
    auto* e = static_cast<Experts*>(PyCapsule_GetPointer(c, kExpertsName));
    if (!e) throw PythonError{};
    return e;
}

// Weights and scales of the shared experts, to be worked on in the same launches (w1, w3, w2).
struct Shared {
    at::Tensor w[3], s[3];
};

// Result of the expert GEMMs of one pass, before the combination: one allocation, carved up.
struct Routed {
    at::Tensor arena, x;
    int64_t T, dim;
    int topk;
    const void *o, *w, *z = nullptr;      // z: the shared experts' output when the pass computed it
    const int32_t* pos;
    // a handful of tokens: w2 and the combination are one launch, still to come
    PyObject* experts = nullptr;          // the capsule, which keeps table and weights
    Shared sh;
    dsv3_few_shared_t few_sh = {};
    const void *route = nullptr, *h = nullptr;
    Routed() = default;
    Routed(const Routed&) = delete;
    ~Routed() { Py_XDECREF(experts); }
};
const char* kRoutedName = "dsv3_b200.routed";
void free_routed(PyObject* c) { delete static_cast<Routed*>(PyCapsule_GetPointer(c, kRoutedName)); }

std::unique_ptr<Routed> run_experts(PyObject* capsule, Experts& e, const at::Tensor& x, const at::Tensor& weights_in, const at::Tensor& indices_in,
                                    int64_t n_routed, bool assume_no_inplace, const Shared* sh) {
    if (indices_in.dim() != 2 || weights_in.sizes() != indices_in.sizes())
        raise(PyExc_ValueError, "routing weights and indices must both be [tokens, top-k]");
    const c10::Device dev = require_cuda(x, weights_in, indices_in, e.table1);
    require(x.is_contiguous(), "Input tensor must be contiguous");     // as act_quant
    if (x.scalar_type() != at::kBFloat16) raise(PyExc_NotImplementedError, "the expert layer takes bfloat16 activations");
    at::Tensor indices = indices_in.scalar_type() == at::kLong ? indices_in : indices_in.to(at::kLong);
    at::Tensor weights = (weights_in.scalar_type() == at::kBFloat16 || weights_in.scalar_type() == at::kFloat) ? weights_in : weights_in.to(at::kFloat);
    if (!indices.is_contiguous()) indices = indices.contiguous();
    if (!weights.is_contiguous()) weights = weights.contiguous();
    const int64_t T = indices.size(0), topk = indices.size(1), P = T * topk, dim = e.dim, inter = e.inter;
    if (x.dim() != 2 || x.size(0) != T || x.size(1) != dim) raise(PyExc_ValueError, "activations must be [tokens, dim]");
    auto r = std::make_unique<Routed>();
    r->T = T;
    r->dim = dim;
    r->topk = static_cast<int>(topk);
    r->x = x;
    // this rank owns n of the layer's experts and, on average, that share of the pairs
    const int64_t hint = n_routed > e.n ? std::max<int64_t>(1, (P * e.n + n_routed - 1) / n_routed) : 0;
    int64_t at = 0;
    auto take = [&](int64_t bytes) {
        const int64_t here = at;
        at += (bytes + 255) & ~int64_t(255);
        return here;
    };
    if (P > 0 && dsv3_few_experts_pay(T, r->topk, e.n, n_routed, dim, inter, sh ? sh->w[0].size(0) : 0)) {
        const int64_t inter_s = sh ? sh->w[0].size(0) : 0;
        const int64_t o_route = take(static_cast<int64_t>(dsv3_few_route_bytes())), o_h = take(2 * P * inter), o_hz = take(2 * T * inter_s);
        r->arena = new_cuda({at}, at::kByte, dev);
        uint8_t* base = static_cast<uint8_t*>(r->arena.data_ptr());
        r->route = base + o_route;
        r->h = base + o_h;
        r->experts = Py_NewRef(capsule);
        if (sh) {
            r->sh = *sh;
            auto scale = [&](int i) { return static_cast<const float*>(sh->s[i].const_data_ptr()); };
            r->few_sh = {sh->w[0].const_data_ptr(), scale(0), sh->w[1].const_data_ptr(), scale(1), sh->w[2].const_data_ptr(), scale(2), inter_s, base + o_hz};
        }
        const void *t1 = e.table1.const_data_ptr(), *t3 = e.table3.const_data_ptr(), *t2 = e.table2.const_data_ptr();
        const void *xp = x.const_data_ptr(), *wp = weights.const_data_ptr();
        const int bf16 = weights.scalar_type() == at::kBFloat16;
        const auto* ip = static_cast<const int64_t*>(indices.const_data_ptr());
        call_library(dev, [&](dsv3_stream_t st) {
            return dsv3_few_up(t1, t3, t2, e.n, xp, T, dim, ip, wp, bf16, r->topk, e.start, inter, e.fmt, base + o_route, base + o_h,
                               sh ? &r->few_sh : nullptr, st);
        });
        return r;
    }
    const int64_t o_seg = take(4 * (e.n + 1)), o_pos = take(4 * P), o_w = take(2 * P), o_xq = take(P * dim), o_xs = take(4 * P * (dim / 128)),
                  o_hq = take(P * inter), o_hs = take(4 * P * (inter / 128)), o_o = take(2 * P * dim);
    const int64_t inter_s = sh ? sh->w[0].size(0) : 0;
    const int64_t o_zh = take(T * inter_s), o_zs = take(4 * T * (inter_s / 128)), o_z = take(sh ? 2 * T * dim : 0);
    r->arena = new_cuda({std::max<int64_t>(at, 1)}, at::kByte, dev);
    uint8_t* base = static_cast<uint8_t*>(r->arena.data_ptr());
    r->o = base + o_o;
    r->w = base + o_w;
    r->pos = reinterpret_cast<const int32_t*>(base + o_pos);
    if (P == 0) return r;
    at::Tensor xq = new_cuda(x.sizes(), at::kFloat8_e4m3fn, dev), xs = new_cuda_last(x, dim / 128, at::kFloat);
    const size_t need = dsv3_gemm_rows_workspace_bytes(e.n, P, hint);
    const at::Tensor held = need ? workspace(dev, need) : at::Tensor();
    void* ws = need ? held.data_ptr() : nullptr;
    const size_t ws_bytes = need ? static_cast<size_t>(held.numel()) : 0;
    auto* seg = reinterpret_cast<int32_t*>(base + o_seg);
    auto* xs_t = reinterpret_cast<float*>(base + o_xs);
    auto* hs_t = reinterpret_cast<float*>(base + o_hs);
    const void *t1 = e.table1.const_data_ptr(), *t3 = e.table3.const_data_ptr(), *t2 = e.table2.const_data_ptr();
    const void *xp = x.const_data_ptr(), *wp = weights.const_data_ptr();
    const int bf16 = weights.scalar_type() == at::kBFloat16;
    const auto* ip = static_cast<const int64_t*>(indices.const_data_ptr());
    void* xqp = xq.data_ptr();
    float* xsp = static_cast<float*>(xs.data_ptr());
    dsv3_side_gemm_t up = {}, down = {};
    if (sh) {
        up = {xqp, xsp, 0, T, inter_s, dim, sh->w[0].const_data_ptr(), static_cast<const float*>(sh->s[0].const_data_ptr()),
              sh->w[1].const_data_ptr(), static_cast<const float*>(sh->s[1].const_data_ptr()), base + o_zh, reinterpret_cast<float*>(base + o_zs)};
        down = {base + o_zh, reinterpret_cast<const float*>(base + o_zs), 1, T, dim, inter_s, sh->w[2].const_data_ptr(),
                static_cast<const float*>(sh->s[2].const_data_ptr()), nullptr, nullptr, base + o_z, nullptr};
        r->z = base + o_z;
    }
    call_library(dev, [&](dsv3_stream_t st) {
        int rc = dsv3_moe_dispatch(xp, T, dim, ip, wp, bf16, r->topk, e.start, e.n, e.fmt, seg, reinterpret_cast<int32_t*>(base + o_pos),
                                   base + o_w, xqp, xsp, base + o_xq, xs_t, st);
        if (rc == DSV3_OK)
            rc = dsv3_expert_gemms(t1, t3, t2, e.n, base + o_xq, xs_t, seg, P, hint, inter, dim, e.fmt, base + o_hq, hs_t, base + o_o,
                                   sh ? &up : nullptr, sh ? &down : nullptr, ws, ws_bytes, st);
        return rc;
    });
    remember(x, 128, e.fmt, assume_no_inplace, xq, xs);
    return r;
}

// ------------------------------------------------------------------ Python entry points
void want_args(Py_ssize_t got, Py_ssize_t want) {
    if (got != want) raise(PyExc_TypeError, "wrong number of arguments");
}

int64_t int_arg(PyObject* o) {
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw PythonError{};
    return v;
}

template <typename F>
PyObject* guarded(F&& f) {
    try {
        return f();
    } catch (const PythonError&) {
        return nullptr;
    } catch (const c10::OutOfMemoryError& e) {
        PyErr_SetString(g_oom_class, e.what_without_backtrace());
        return nullptr;
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

PyObject* py_set_error_class(PyObject*, PyObject* cls) {
    Py_XSETREF(g_error_class, Py_NewRef(cls));
    Py_RETURN_NONE;
}

PyObject* py_act_quant(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        want_args(n, 3);
        auto r = quantise(tensor_arg(args[0]), int_arg(args[1]), scale_fmt_arg(args[2]));
        return wrap_pair(std::move(r.first), std::move(r.second));
    });
}

PyObject* py_swiglu_quant(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        want_args(n, 3);
        const at::Tensor &a = tensor_arg(args[0]), &b = tensor_arg(args[1]);
        const int fmt = scale_fmt_arg(args[2]);
        require(a.is_contiguous() && b.is_contiguous(), "Input tensors must be contiguous");
        const int64_t K = last_dim(a);
        require(a.sizes() == b.sizes() && K % 128 == 0, "a and b must have the same shape, last dimension divisible by 128");
        const c10::Device dev = require_cuda(a, b);
        if (a.scalar_type() != at::kBFloat16 || b.scalar_type() != at::kBFloat16)
            raise(PyExc_NotImplementedError, "swiglu_quant takes bfloat16 tensors");
        const int64_t rows = K ? a.numel() / K : 0;
        at::Tensor y = new_cuda(a.sizes(), at::kFloat8_e4m3fn, dev);
        at::Tensor s = new_cuda_last(a, K / 128, at::kFloat);
        const void *ap = a.const_data_ptr(), *bp = b.const_data_ptr();
        void* yp = y.data_ptr();
        float* sp = static_cast<float*>(s.data_ptr());
        call_library(dev, [&](dsv3_stream_t st) { return dsv3_swiglu_quant(ap, bp, rows, K, fmt, yp, sp, st); });
        return wrap_pair(std::move(y), std::move(s));
    });
}

PyObject* py_weight_dequant(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        want_args(n, 3);
        const at::Tensor &x = tensor_arg(args[0]), &s = tensor_arg(args[1]);
        const int64_t block = int_arg(args[2]);
        require(x.is_contiguous() && s.is_contiguous(), "Input tensors must be contiguous");
        require(x.dim() == 2 && s.dim() == 2, "Input tensors must have 2 dimensions");
        const c10::Device dev = require_cuda(x, s);
        if (x.element_size() != 1 || s.scalar_type() != at::kFloat)
            raise(PyExc_NotImplementedError, "weight_dequant takes a 1-byte FP8 weight and float32 scales");
        require_bf16_default();
        at::Tensor y = new_cuda(x.sizes(), at::kBFloat16, dev);
        const int64_t N = x.size(0), K = x.size(1);
        const void* xp = x.const_data_ptr();
        const float* sp = static_cast<const float*>(s.const_data_ptr());
        void* yp = y.data_ptr();
        call_library(dev, [&](dsv3_stream_t st) { return dsv3_weight_dequant(xp, sp, N, K, static_cast<int>(block), yp, st); });
        return wrap(std::move(y));
    });
}

PyObject* py_fp8_gemm(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        want_args(n, 4);
        return wrap(gemm(tensor_arg(args[0]), tensor_arg(args[1]), tensor_arg(args[2]), tensor_arg(args[3])));
    });
}

PyObject* py_fp8_linear(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        want_args(n, 4);
        return wrap(linear_small(tensor_arg(args[0]), tensor_arg(args[1]), tensor_arg(args[2]), scale_fmt_arg(args[3])));
    });
}

// (x, weight, block_size, scale_fmt, assume_no_inplace, fused_max_rows, fused_max_bytes, fused_max_bytes_3_rows): linear()'s FP8
// branch.  The limits of the fused launch, with their reasons, are in ops.py.
PyObject* py_linear(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        want_args(n, 8);
        const at::Tensor &x = tensor_arg(args[0]), &w = tensor_arg(args[1]);
        const int64_t block = int_arg(args[2]);
        const int fmt = scale_fmt_arg(args[3]);
        PyObject* scale_obj = PyObject_GetAttr(args[1], g_attr_scale);
        if (!scale_obj) throw PythonError{};
        at::Tensor scale;
        if (THPVariable_Check(scale_obj)) scale = THPVariable_Unpack(scale_obj);
        Py_DECREF(scale_obj);
        if (!scale.defined()) raise(PyExc_TypeError, "weight.scale is not a tensor");
        const int64_t K = last_dim(x), rows = K ? x.numel() / K : 0;
        if (rows > 0 && rows <= int_arg(args[5]) && w.numel() <= int_arg(args[rows <= 2 ? 6 : 7]) && block == 128 && K % 128 == 0 &&
            x.scalar_type() == at::kBFloat16 && x.is_contiguous()) {
            count(g_key_fused);
            return wrap(linear_small(x, w, scale, fmt));
        }
        auto q = quantise_remembered(x, block, fmt, PyObject_IsTrue(args[4]) == 1);
        return wrap(gemm(q.first, q.second, w, scale));
    });
}

// (x, w1, w3, w2, scale_fmt of x, scale_fmt in front of w2, assume_no_inplace) -> y, or None where the separate launches are faster
PyObject* py_mlp(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        want_args(n, 7);
        at::Tensor w[3], s[3];
        for (int i = 0; i < 3; ++i) {
            w[i] = tensor_arg(args[1 + i]);
            PyObject* scale_obj = PyObject_GetAttr(args[1 + i], g_attr_scale);
            if (!scale_obj) throw PythonError{};
            if (THPVariable_Check(scale_obj)) s[i] = THPVariable_Unpack(scale_obj);
            Py_DECREF(scale_obj);
            if (!s[i].defined()) raise(PyExc_TypeError, "weight.scale is not a tensor");
        }
        at::Tensor y = mlp(tensor_arg(args[0]), w, s, scale_fmt_arg(args[4]), scale_fmt_arg(args[5]), PyObject_IsTrue(args[6]) == 1);
        if (!y.defined()) Py_RETURN_NONE;
        return wrap(std::move(y));
    });
}

// Whether a call of any of these objects does more than its class's forward: hooks, a forward of its own, a compiled call.  (Here, as
// four are asked about per call of an expert layer: 0.2 us together instead of 0.15 each.)
PyObject* py_intercepted(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        int found = 0;
        for (Py_ssize_t i = 0; i < n && found == 0; ++i) {
            PyObject* own = PyObject_GetAttr(args[i], g_attr_dict);
            if (!own) {
                if (!PyErr_ExceptionMatches(PyExc_AttributeError)) throw PythonError{};
                PyErr_Clear();
                continue;
            }
            found = 1;
            if (PyDict_Check(own)) {
                const auto at = [&](PyObject* key) { return PyDict_GetItemWithError(own, key); };
                PyObject* compiled = at(g_key_compiled);
                found = at(g_key_forward) != nullptr || (compiled && compiled != Py_None);
                for (PyObject* key : {g_key_hooks, g_key_pre_hooks}) {
                    PyObject* hooks = found ? nullptr : at(key);
                    if (hooks) found = PyObject_IsTrue(hooks);
                }
            }
            Py_DECREF(own);
        }
        if (found < 0 || PyErr_Occurred()) throw PythonError{};
        return PyBool_FromLong(found);
    });
}

// (w1, w3, w2): FP8 weights whose products can be quantised together in front of w2
PyObject* py_fp8_weights(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        want_args(n, 3);
        for (int i = 0; i < 3; ++i)
            if (!THPVariable_Check(args[i]) || THPVariable_Unpack(args[i]).element_size() != 1) Py_RETURN_FALSE;
        const at::Tensor& w2 = THPVariable_Unpack(args[2]);
        return PyBool_FromLong(w2.dim() > 1 && w2.size(1) % 128 == 0);
    });
}

// (x, block_size, scale_fmt, assume_no_inplace) -> (y, s), remembered
PyObject* py_quantise_remembered(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        want_args(n, 4);
        auto r = quantise_remembered(tensor_arg(args[0]), int_arg(args[1]), scale_fmt_arg(args[2]), PyObject_IsTrue(args[3]) == 1);
        return wrap_pair(std::move(r.first), std::move(r.second));
    });
}

// (n, start, dim, inter, scale_fmt, table1, table3, table2, list or None, members, look-ups [(dict, key, value)], weights and
// scales)
PyObject* py_experts(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        want_args(n, 12);
        auto e = std::make_unique<Experts>();
        e->list = nullptr;
        e->n = static_cast<int>(int_arg(args[0]));
        e->start = static_cast<int>(int_arg(args[1]));
        e->dim = int_arg(args[2]);
        e->inter = int_arg(args[3]);
        e->fmt = scale_fmt_arg(args[4]);
        e->table1 = tensor_arg(args[5]);
        e->table3 = tensor_arg(args[6]);
        e->table2 = tensor_arg(args[7]);
        if (PyList_Check(args[8])) e->list = Py_NewRef(args[8]);
        if (!PyList_Check(args[9]) || !PyList_Check(args[10]) || !PyList_Check(args[11]) || PyList_GET_SIZE(args[9]) != e->n)
            raise(PyExc_TypeError, "members, look-ups and tensors are lists");
        for (Py_ssize_t i = 0; i < PyList_GET_SIZE(args[9]); ++i) e->members.push_back(Py_NewRef(PyList_GET_ITEM(args[9], i)));
        for (Py_ssize_t i = 0; i < PyList_GET_SIZE(args[10]); ++i) {
            PyObject *d, *k, *v;
            if (!PyArg_ParseTuple(PyList_GET_ITEM(args[10], i), "O!OO", &PyDict_Type, &d, &k, &v)) throw PythonError{};
            e->lookups.push_back({Py_NewRef(d), Py_NewRef(k), Py_NewRef(v)});
#if PY_VERSION_HEX >= 0x030C0000
            if (g_watcher >= 0 && PyDict_Watch(g_watcher, d) != 0) throw PythonError{};
#endif
        }
        for (Py_ssize_t i = 0; i < PyList_GET_SIZE(args[11]); ++i) {
            PyObject* t = PyList_GET_ITEM(args[11], i);
            const void* at = tensor_arg(t).const_data_ptr();
            e->tensors.emplace_back(Py_NewRef(t), at);
        }
        return PyCapsule_New(e.release(), kExpertsName, free_experts);
    });
}

PyObject* py_experts_current(PyObject*, PyObject* capsule) {
    return guarded([&]() -> PyObject* { return PyBool_FromLong(experts_arg(capsule)->current()); });
}

// (experts, x, weights, indices, n_routed, assume_no_inplace, shared or None) -> result to hand to `combine`
// shared: (w1, w3, w2) weights with their scales as attributes
PyObject* py_run_experts(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        want_args(n, 7);
        Experts& e = *experts_arg(args[0]);
        Shared sh;
        const bool with_shared = args[6] != Py_None;
        if (with_shared) {
            if (!PyTuple_Check(args[6]) || PyTuple_GET_SIZE(args[6]) != 3) raise(PyExc_TypeError, "shared is a tuple of three weights");
            for (int i = 0; i < 3; ++i) {
                PyObject* w = PyTuple_GET_ITEM(args[6], i);
                sh.w[i] = tensor_arg(w);
                PyObject* sc = PyObject_GetAttr(w, g_attr_scale);
                if (!sc) throw PythonError{};
                if (THPVariable_Check(sc)) sh.s[i] = THPVariable_Unpack(sc);
                Py_DECREF(sc);
                if (!sh.s[i].defined() || !sh.w[i].is_contiguous() || !sh.s[i].is_contiguous() || sh.s[i].scalar_type() != at::kFloat)
                    raise(PyExc_ValueError, "shared weights and scales must be contiguous, scales float32");
            }
            require_cuda(e.table1, sh.w[0], sh.w[1], sh.w[2], sh.s[0], sh.s[1], sh.s[2]);
            const int64_t f = sh.w[0].size(0);
            if (sh.w[0].size(1) != e.dim || sh.w[1].sizes() != sh.w[0].sizes() || sh.w[2].size(0) != e.dim || sh.w[2].size(1) != f || f % 128 != 0)
                raise(PyExc_ValueError, "shared weights do not fit the layer");
        }
        auto r = run_experts(args[0], e, tensor_arg(args[1]), tensor_arg(args[2]), tensor_arg(args[3]), int_arg(args[4]),
                             PyObject_IsTrue(args[5]) == 1, with_shared ? &sh : nullptr);
        return PyCapsule_New(r.release(), kRoutedName, free_routed);
    });
}

// Whether w2 of this pass is still to come (with the combination): until then its weights must stay what they were.
PyObject* py_weights_pending(PyObject*, PyObject* routed) {
    return guarded([&]() -> PyObject* {
        auto* r = static_cast<Routed*>(PyCapsule_GetPointer(routed, kRoutedName));
        if (!r) throw PythonError{};
        return PyBool_FromLong(r->route != nullptr);
    });
}

// (result of run_experts, z or None): the tokens' weighted sums, plus z (or the shared experts' output computed along)
PyObject* py_combine(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        want_args(n, 2);
        auto* r = static_cast<Routed*>(PyCapsule_GetPointer(args[0], kRoutedName));
        if (!r) throw PythonError{};
        const c10::Device dev = r->arena.device();
        const void* zp = r->z;
        if (args[1] != Py_None) {
            const at::Tensor& z = tensor_arg(args[1]);
            if (!z.is_contiguous() || z.scalar_type() != at::kBFloat16 || z.device() != dev || z.numel() != r->T * r->dim)
                raise(PyExc_ValueError, "z must be a contiguous bfloat16 tensor of the layer's output size on the same device");
            zp = z.const_data_ptr();
        }
        at::Tensor y = new_cuda({r->T, r->dim}, at::kBFloat16, dev);
        void* yp = y.data_ptr();
        if (r->route) {
            const bool own = r->sh.w[0].defined() && args[1] == Py_None;       // z takes the place of what was computed along
            const Experts& e = *experts_arg(r->experts);
            const void* t2 = e.table2.const_data_ptr();
            call_library(dev, [&](dsv3_stream_t st) {
                return dsv3_few_down(t2, e.n, r->route, r->h, r->T, r->topk, r->dim, e.inter, e.fmt, own ? &r->few_sh : nullptr, zp, yp, st);
            });
            return wrap(std::move(y));
        }
        call_library(dev, [&](dsv3_stream_t st) { return dsv3_moe_combine_add(r->o, r->pos, r->w, zp, r->T, r->topk, r->dim, yp, st); });
        return wrap(std::move(y));
    });
}

PyObject* py_set_stats(PyObject*, PyObject* dict) {
    Py_XSETREF(g_stats, Py_NewRef(dict));
    Py_RETURN_NONE;
}

PyObject* py_forget(PyObject*, PyObject*) {
    g_memo.clear();
    Py_RETURN_NONE;
}

// After a bounded wait gave up, tickets may be left non-zero: the next call gets a new workspace with a clear header.  (A
// workspace is not cleared in place: its stream may be in a capture, or gone.  A graph clears its own at every replay.)
PyObject* py_drop_workspaces(PyObject*, PyObject*) {
    g_workspaces.clear();
    Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"set_error_class", py_set_error_class, METH_O, "class raised for a non-zero status: cls(status, message)"},
    {"act_quant", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_act_quant)), METH_FASTCALL, "(x, block_size, scale_fmt)"},
    {"swiglu_quant", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_swiglu_quant)), METH_FASTCALL, "(a, b, scale_fmt)"},
    {"weight_dequant", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_weight_dequant)), METH_FASTCALL, "(x, s, block_size)"},
    {"fp8_gemm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_fp8_gemm)), METH_FASTCALL, "(a, a_s, b, b_s)"},
    {"fp8_linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_fp8_linear)), METH_FASTCALL, "(x, weight, scale, scale_fmt)"},
    {"linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_linear)), METH_FASTCALL,
     "(x, weight, block_size, scale_fmt, assume_no_inplace, fused_max_rows, fused_max_bytes, fused_max_bytes_3_rows)"},
    {"mlp", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_mlp)), METH_FASTCALL, "(x, w1, w3, w2, x_fmt, h_fmt, assume_no_inplace)"},
    {"intercepted", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_intercepted)), METH_FASTCALL,
     "whether a call of any of these objects does more than its class's forward"},
    {"fp8_weights", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_fp8_weights)), METH_FASTCALL, "(w1, w3, w2)"},
    {"quantise_remembered", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_quantise_remembered)), METH_FASTCALL,
     "(x, block_size, scale_fmt, assume_no_inplace)"},
    {"experts", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_experts)), METH_FASTCALL,
     "(n, start, dim, inter, scale_fmt, table1, table3, table2, list, members, lookups, tensors)"},
    {"experts_current", py_experts_current, METH_O, "whether the experts are still those the tables were built from"},
    {"run_experts", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_run_experts)), METH_FASTCALL,
     "(experts, x, weights, indices, n_routed, assume_no_inplace, shared)"},
    {"weights_pending", py_weights_pending, METH_O, "whether `combine` of this result still reads the experts' weights"},
    {"combine", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_combine)), METH_FASTCALL, "(routed, z)"},
    {"set_stats", py_set_stats, METH_O, "dict whose counters linear() keeps"},
    {"forget", py_forget, METH_NOARGS, "drop the remembered quantisations"},
    {"drop_workspaces", py_drop_workspaces, METH_NOARGS, "give the split-K workspaces back"},
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_dsv3_host", "Native host path of the dsv3_b200 operators.", -1, methods,
                          nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__dsv3_host(void) {
    g_key_calls = PyUnicode_InternFromString("act_quant_calls");
    g_key_reused = PyUnicode_InternFromString("act_quant_reused");
    g_key_fused = PyUnicode_InternFromString("fused_linear_calls");
    g_attr_scale = PyUnicode_InternFromString("scale");
    g_attr_dict = PyUnicode_InternFromString("__dict__");
    g_key_forward = PyUnicode_InternFromString("forward");
    g_key_hooks = PyUnicode_InternFromString("_forward_hooks");
    g_key_pre_hooks = PyUnicode_InternFromString("_forward_pre_hooks");
    g_key_compiled = PyUnicode_InternFromString("_compiled_call_impl");
#if PY_VERSION_HEX >= 0x030C0000
    g_watcher = PyDict_AddWatcher(on_dict_change);
    if (g_watcher < 0) PyErr_Clear();       // all watchers taken: look-ups are verified on every pass
#endif
    PyObject* torch = PyImport_ImportModule("torch");
    g_oom_class = torch ? PyObject_GetAttrString(torch, "OutOfMemoryError") : nullptr;
    Py_XDECREF(torch);
    if (!g_oom_class) return nullptr;
    for (PyObject* name : {g_key_calls, g_key_reused, g_key_fused, g_attr_scale, g_attr_dict, g_key_forward, g_key_hooks, g_key_pre_hooks, g_key_compiled})
        if (!name) return nullptr;
    return PyModule_Create(&module_def);
}
