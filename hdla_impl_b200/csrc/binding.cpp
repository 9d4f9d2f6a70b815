// Native host path between PyTorch and libhdla: argument checks, allocation, autograd nodes and the status protocol of
// the entry points, in one call from Python.  A small call of the operator is bound by this host work, not by its
// kernels: through ctypes and Python autograd functions a decode step of 64 heads took 36 us of which 6 were the
// kernel, and a training step of 32 chunk tiles 355 us.
//
// Every function here takes the ordinary case -- plain CUDA tensors with consistent shapes and types -- and answers
// NotImplemented to anything else; the Python wrapper then takes its own route, which raises the errors.  The kernels
// are reached through the C ABI of include/hdla.h only (bind() looks its functions up in the loaded library).
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime.h>
#include <dlfcn.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/grad_mode.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <atomic>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/hdla.h"
#include "status_board.h"

namespace {

using at::Tensor;

// ------------------------------------------------------------------------------------------ C ABI
struct Abi {
    decltype(&hdla_chunk_workspace_bytes) workspace_bytes;
    decltype(&hdla_chunk_uses_tensor_cores) uses_tensor_cores;
    decltype(&hdla_fp32_status_words) fp32_status_words;
    decltype(&hdla_chunk_fwd) chunk_fwd;
    decltype(&hdla_chunk_bwd) chunk_bwd;
    decltype(&hdla_recurrent_fwd) recurrent_fwd;
    decltype(&hdla_norm_gate_fwd) norm_gate_fwd;
    decltype(&hdla_norm_gate_bwd) norm_gate_bwd;
    decltype(&hdla_last_error) last_error;
} abi{};

template <typename F>
void look_up(void* handle, const char* name, F& f) {
    f = reinterpret_cast<F>(dlsym(handle, name));
    if (!f) throw std::runtime_error(std::string("libhdla has no ") + name);
}

void check(int rc, const char* what) {
    if (rc != 0) throw std::runtime_error(std::string(what) + " failed (code " + std::to_string(rc) + "): " + abi.last_error());
}

void check_cuda(cudaError_t e, const char* what) {
    if (e != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
}

bool env_is_1(const char* name) {
    const char* v = getenv(name);
    return v && v[0] == '1' && v[1] == 0;
}

// ------------------------------------------------------------------------------------------ small helpers
// A plain tensor (torch.Tensor or nn.Parameter itself: subclasses have their own dispatch).
bool plain(PyObject* o) {
    return THPVariable_CheckExact(o) || (ParameterClass && Py_TYPE(o) == reinterpret_cast<PyTypeObject*>(ParameterClass));
}
const Tensor* as_tensor(PyObject* o) { return plain(o) ? &THPVariable_Unpack(o) : nullptr; }

int dtype_code(const Tensor& t) {
    const auto s = t.scalar_type();
    return s == at::kFloat ? HDLA_F32 : s == at::kBFloat16 ? HDLA_BF16 : -1;
}
const void* ptr(const Tensor& t) { return t.defined() ? t.const_data_ptr() : nullptr; }
void* mptr(const Tensor& t) { return t.defined() ? t.mutable_data_ptr() : nullptr; }
float* fptr(const Tensor& t) { return t.defined() ? static_cast<float*>(t.mutable_data_ptr()) : nullptr; }

Tensor dense(at::IntArrayRef size, at::ScalarType st, const at::Device& dev) {
    return at::detail::empty_cuda(size, st, dev, std::nullopt);
}
Tensor dense_like(const Tensor& t) { return dense(t.sizes(), t.scalar_type(), t.device()); }
Tensor f32_contiguous(const Tensor& t) { return t.defined() ? t.to(at::kFloat).contiguous() : t; }

bool transforms_active() {        // functorch transforms wrap tensors; the Python route says that they are not supported
    return c10::impl::tls_local_dispatch_key_set().included_.has(c10::DispatchKey::FuncTorchDynamicLayerFrontMode);
}
// A tracer records the Python autograd functions as calls (inside which it may go on tracing); of what happens here it
// would see nothing but tensors out of nowhere.
bool tracing() { return torch::jit::tracer::isTracing(); }
bool capturing(cudaStream_t st) {
    cudaStreamCaptureStatus s = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(st, &s) == cudaSuccess && s != cudaStreamCaptureStatusNone;
}

PyObject* wrap(const Tensor& t) {
    if (!t.defined()) Py_RETURN_NONE;
    return THPVariable_Wrap(t);
}

// ------------------------------------------------------------------------------------------ status protocol
// The bf16 kernels report in the first words of the workspace: word 0 a device-side wait that ran out, word 1 a chunk
// whose log decay is beyond what that pipeline represents, word 2 the largest chunk decay of the call.  After every
// call the words are copied to pinned host memory without blocking and looked at the next time the device is used.
//
// A decay overflow is different from the other conditions: the call's results are wrong but the fp32 pipeline would
// have computed them correctly.  Forward therefore WAITS for its own status words -- and reruns the call on the fp32
// pipeline when word 1 is set -- whenever an overflow is plausible: on the first call on a device, and from then on
// while the largest chunk decay seen on that device is above half the limit.  HDLA_STRICT=1 always waits;
// HDLA_ASYNC_STATUS=1 never does (an overflow then raises at the next entry).
//
// A call that is captured into a graph posts nothing: its copy would land at every replay, when no caller waits for it
// and the slot may be another call's.
//
// Backward runs on autograd's own threads without the GIL: the boards have locks of their own, which are not held while
// an event is waited for or Python code runs.
constexpr double kDecayLimit = 150.0;
struct Gpu {                                  // what status_board.h asks for
    typedef cudaEvent_t Event;
    typedef cudaStream_t Stream;
    static int32_t* alloc_words(int slots) {
        void* p = nullptr;
        check_cuda(cudaHostAlloc(&p, static_cast<size_t>(slots) * 16, cudaHostAllocPortable), "status words");
        return static_cast<int32_t*>(p);
    }
    static Event make_event(int dev) {
        c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(dev));
        cudaEvent_t e;
        check_cuda(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "status event");
        return e;
    }
    static void copy(int32_t* dst, const void* src, Stream st) {
        check_cuda(cudaMemcpyAsync(dst, src, 16, cudaMemcpyDeviceToHost, st), "status words");
    }
    static void record(Event e, Stream st) { check_cuda(cudaEventRecord(e, st), "status words"); }
    static bool done(Event e) {
        const cudaError_t r = cudaEventQuery(e);
        if (r == cudaErrorNotReady) { cudaGetLastError(); return false; }
        check_cuda(r, "status words");
        return true;
    }
    static void wait(Event e) {
        cudaError_t r;
        if (PyGILState_Check()) {
            Py_BEGIN_ALLOW_THREADS
            r = cudaEventSynchronize(e);
            Py_END_ALLOW_THREADS
        } else {
            r = cudaEventSynchronize(e);
        }
        check_cuda(r, "status words");
    }
};
typedef hdla_host::StatusBoard<Gpu> Board;

[[noreturn]] void status_fail(const int32_t* w) {
    if (w[0])
        throw std::runtime_error("libhdla: a device-side wait ran out (code " + std::to_string(w[0]) +
                                 "); the results of that call are invalid");
    throw std::runtime_error(
        "libhdla: the total log decay of some chunk exceeds 150 in some channel, beyond what the bf16 tensor-core "
        "pipeline represents; the results of that call are invalid. Set HDLA_FORCE_SIMT=1 to use the fp32 pipeline, "
        "which has no such limit.");
}
struct DeviceState {
    Board board;
    std::atomic<unsigned> fp32_calls{0};
    explicit DeviceState(int dev) : board(dev, status_fail) {}
};
std::map<int, DeviceState> g_devices;         // by device; an entry stays where it is
std::mutex g_mu;
typedef std::unique_lock<std::mutex> Lock;

DeviceState& state_of(int dev) {
    Lock lk(g_mu);
    return g_devices.try_emplace(dev, dev).first->second;
}
Board& board_of(int dev) { return state_of(dev).board; }

// The fp32 pipeline's kernels have one set of words per device, written only when a wait has run out.  A training step there
// can take less time than copying words after every call would: every kFp32Every-th call posts them, and so does a check
// that waits.
constexpr unsigned kFp32Every = 64;
void fp32_post(int dev, cudaStream_t stream) {
    void* words = nullptr;
    check(abi.fp32_status_words(&words), "hdla_fp32_status_words");
    Board& board = board_of(dev);
    board.publish(board.post(words, stream));
}
// Look at the words that have landed (with `wait`, at all of them); throws if one reports a problem.
void status_check(int dev, bool wait) {
    if (wait && state_of(dev).fp32_calls != 0) {
        c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(dev));
        check_cuda(cudaDeviceSynchronize(), "status words");
        fp32_post(dev, c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(dev)).stream());
    }
    board_of(dev).check(wait);
}
void fp32_called(int dev, cudaStream_t stream, bool is_capturing) {
    if (is_capturing) return;
    const unsigned calls = ++state_of(dev).fp32_calls;
    if (env_is_1("HDLA_STRICT")) status_check(dev, true);
    else if (calls % kFp32Every == 0) fp32_post(dev, stream);
}
void status_post(const void* ws, int dev, cudaStream_t stream, bool is_capturing) {
    if (is_capturing) return;
    Board& board = board_of(dev);
    board.publish(board.post(ws, stream));
    if (env_is_1("HDLA_STRICT")) board.check(true);
}
bool overflow_plausible(Board& board) {
    if (env_is_1("HDLA_ASYNC_STATUS")) return false;
    if (env_is_1("HDLA_STRICT")) return true;
    const double decay = board.decay();
    return decay != decay || decay > 0.5 * kDecayLimit;
}

// ------------------------------------------------------------------------------------------ chunked operator
struct DecayOverflow {};          // the caller has another route for a decay beyond the bf16 pipeline

struct ChunkArgs {
    HdlaDims d{};
    std::vector<int64_t> cu;      // offsets of a packed batch (empty: uniform)
    int n_states = 0;
    double scale = 1.0;
    HdlaDims dims(int extra = 0) const {
        HdlaDims x = d;
        x.flags |= extra;
        if (!cu.empty()) { x.cu_seqlens = cu.data(); x.n_seqs = static_cast<int>(cu.size()) - 1; }
        return x;
    }
};

bool tc_shape(const Tensor& q, int64_t T, int64_t K, int64_t V, int64_t R) {
    return q.scalar_type() == at::kBFloat16 && R == 2 && K % 8 == 0 && V % 8 == 0 && K >= 8 && K <= 128 && V >= 8 &&
           V <= 128 && T > 32;
}

struct ChunkOut { Tensor o, ht, ws; bool forced_simt = false; };

// One forward call on contiguous tensors.  `a` is beta and `b` undefined with HDLA_FLAG_PARAM_AB.
ChunkOut chunk_forward(const ChunkArgs& c, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& a,
                       const Tensor& b, const Tensor& gk, const Tensor& h0, bool want_ht, bool keep_ws, bool force_simt) {
    const int dev = q.get_device();
    c10::cuda::CUDAGuard guard(q.device());
    const cudaStream_t st = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(dev)).stream();
    const bool cap = capturing(st);
    if (!cap) status_check(dev, false);
    const HdlaDims d = c.dims(force_simt ? HDLA_FLAG_FORCE_SIMT : 0);
    const size_t n = abi.workspace_bytes(&d, keep_ws ? 1 : 0);
    if (n == 0) throw std::runtime_error(std::string("unsupported problem: ") + abi.last_error());
    ChunkOut r;
    r.forced_simt = force_simt;
    r.ws = dense({static_cast<int64_t>(n)}, at::kByte, q.device());
    r.o = dense_like(v);
    if (want_ht) r.ht = dense({c.n_states, d.H, d.K, d.V}, at::kFloat, q.device());
    check(abi.chunk_fwd(&d, ptr(q), ptr(k), ptr(v), ptr(a), ptr(b), ptr(gk), static_cast<float>(c.scale), fptr(h0),
                        mptr(r.o), fptr(r.ht), mptr(r.ws), n, st), "hdla_chunk_fwd");
    if (abi.uses_tensor_cores(&d)) {
        Board& board = board_of(dev);
        if (!cap && overflow_plausible(board)) {
            int32_t w[4];
            board.take(board.post(ptr(r.ws), st), w);
            // (the fp32 pipeline takes no packed batches: the caller's per-sequence path has to be used for such decays)
            if (w[1] && !w[0] && (c.cu.empty() || (d.flags & HDLA_FLAG_PARAM_AB))) throw DecayOverflow();
            if (w[0] || w[1]) status_fail(w);
        } else {
            status_post(ptr(r.ws), dev, st, cap);
        }
    } else {
        fp32_called(dev, st, cap);
    }
    if (!keep_ws) r.ws = Tensor();
    return r;
}

struct ChunkGrads { Tensor dq, dk, dv, da, db, dgk, dh0; };

ChunkGrads chunk_backward(const ChunkArgs& c, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& a,
                          const Tensor& b, const Tensor& gk, const Tensor& h0, Tensor d_o, Tensor dht, Tensor ws,
                          bool force_simt) {
    const int dev = q.get_device();
    c10::cuda::CUDAGuard guard(q.device());
    const cudaStream_t st = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(dev)).stream();
    const bool cap = capturing(st);
    if (!cap) status_check(dev, false);
    const HdlaDims d = c.dims((force_simt ? HDLA_FLAG_FORCE_SIMT : 0) | (ws.defined() ? HDLA_FLAG_WS_HOLDS_FWD : 0));
    d_o = d_o.defined() ? d_o.to(q.scalar_type()).contiguous() : at::zeros(v.sizes(), v.options());
    dht = f32_contiguous(dht);
    if (!ws.defined()) {
        const size_t n = abi.workspace_bytes(&d, 1);
        if (n == 0) throw std::runtime_error(std::string("unsupported problem: ") + abi.last_error());
        ws = dense({static_cast<int64_t>(n)}, at::kByte, q.device());
    }
    ChunkGrads g;
    g.dq = dense_like(q); g.dk = dense_like(k); g.dv = dense_like(v); g.da = dense_like(a); g.dgk = dense_like(gk);
    if (b.defined()) g.db = dense_like(b);
    if (h0.defined()) g.dh0 = dense_like(h0);
    check(abi.chunk_bwd(&d, ptr(q), ptr(k), ptr(v), ptr(a), ptr(b), ptr(gk), static_cast<float>(c.scale), fptr(h0),
                        ptr(d_o), fptr(dht), mptr(g.dq), mptr(g.dk), mptr(g.dv), mptr(g.da), mptr(g.db), mptr(g.dgk),
                        fptr(g.dh0), mptr(ws), static_cast<size_t>(ws.numel()), st), "hdla_chunk_bwd");
    if (abi.uses_tensor_cores(&d)) status_post(ptr(ws), dev, st, cap);
    else fp32_called(dev, st, cap);
    return g;
}

PyObject* g_on_overflow = nullptr;        // Python callable: warns (once) that a call is rerun on the fp32 pipeline
struct PythonError {};                    // a Python exception is set

void warn_overflow() {
    PyGILState_STATE gs = PyGILState_Ensure();
    PyObject* r = g_on_overflow ? PyObject_CallNoArgs(g_on_overflow) : nullptr;
    const bool bad = !r && PyErr_Occurred();
    Py_XDECREF(r);
    PyGILState_Release(gs);
    if (bad) throw PythonError();
}

// the forward call, rerun on the fp32 pipeline where the decay asks for it and the operator has that route itself
ChunkOut chunk_forward_any(const ChunkArgs& c, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& a,
                           const Tensor& b, const Tensor& gk, const Tensor& h0, bool want_ht, bool keep_ws) {
    try {
        return chunk_forward(c, q, k, v, a, b, gk, h0, want_ht, keep_ws, false);
    } catch (const DecayOverflow&) {
        if (c.d.flags & HDLA_FLAG_PARAM_AB) throw;
    }
    warn_overflow();
    return chunk_forward(c, q, k, v, a, b, gk, h0, want_ht, keep_ws, true);
}

// ------------------------------------------------------------------------------------------ autograd nodes
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

bool needs_grad(std::initializer_list<const Tensor*> ts) {
    if (!at::GradMode::is_enabled()) return false;
    for (const Tensor* t : ts)
        if (t->defined() && t->requires_grad()) return true;
    return false;
}

// A saved contiguous tensor.  What a saved-tensor hook hands back is looked at before a kernel gets its pointer.
struct Saved {
    SavedVariable var;
    std::vector<int64_t> size;
    at::ScalarType type = at::kFloat;
    at::Device device = at::kCPU;
    bool defined = false;

    void save(const Tensor& t) {
        var = SavedVariable(t, false);
        defined = t.defined();
        if (defined) { size = t.sizes().vec(); type = t.scalar_type(); device = t.device(); }
    }
    Tensor get(const char* node) const {
        const Tensor t = var.unpack();
        if (!defined) return t;
        if (!t.defined() || t.device() != device || t.scalar_type() != type || t.sizes() != at::IntArrayRef(size) ||
            t.layout() != at::kStrided)
            throw std::runtime_error(std::string(node) + ": a saved-tensor hook returned a tensor of another shape, type or "
                                     "device than the saved one's");
        return t.contiguous();
    }
};

template <typename NodeT>
std::shared_ptr<NodeT> make_node() { return std::shared_ptr<NodeT>(new NodeT(), torch::autograd::deleteNode); }

// Saves the inputs and, by default, the forward workspace.  A second backward through the same graph (retain_graph) finds
// the workspace gone -- the backward kernels write into it -- and recomputes what it held.
struct ChunkNode : torch::autograd::Node {
    ChunkArgs args;
    Saved q, k, v, a, b, gk, h0;
    Tensor ws;
    bool force_simt = false;
    at::ScalarType a_type, h0_type;

    std::string name() const override { return "HdlaChunkBackward"; }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (Saved* s : {&q, &k, &v, &a, &b, &gk, &h0}) s->var.reset_data();
        ws = Tensor();
    }
    variable_list apply(variable_list&& grads) override {
        std::lock_guard<std::mutex> lock(mutex_);
        at::NoGradGuard no_grad;
        if (!grads[0].defined() && (grads.size() < 2 || !grads[1].defined())) return variable_list(7);
        Tensor w = std::move(ws);
        ws = Tensor();
        const char* me = "HdlaChunkBackward";
        ChunkGrads g = chunk_backward(args, q.get(me), k.get(me), v.get(me), a.get(me), b.get(me), gk.get(me), h0.get(me),
                                      grads[0], grads.size() > 1 ? grads[1] : Tensor(), std::move(w), force_simt);
        if (g.da.scalar_type() != a_type) g.da = g.da.to(a_type);
        if (g.dh0.defined() && g.dh0.scalar_type() != h0_type) g.dh0 = g.dh0.to(h0_type);
        return {g.dq, g.dk, g.dv, g.da, g.db, g.dgk, g.dh0};
    }
};

// The operator with its gradient: (o, final state or undefined).
std::pair<Tensor, Tensor> chunk_op(const ChunkArgs& args, const Tensor& q_, const Tensor& k_, const Tensor& v_,
                                   const Tensor& a_, const Tensor& b_, const Tensor& gk_, const Tensor& h0_, bool want_ht) {
    const bool grad = needs_grad({&q_, &k_, &v_, &a_, &b_, &gk_, &h0_});
    ChunkOut r;
    std::shared_ptr<ChunkNode> node;
    {
        at::NoGradGuard no_grad;
        const Tensor q = q_.contiguous(), k = k_.contiguous(), v = v_.contiguous(), gk = gk_.contiguous();
        const Tensor a = a_.to(q.scalar_type()).contiguous(), b = b_.defined() ? b_.contiguous() : b_;
        const Tensor h0 = f32_contiguous(h0_);
        r = chunk_forward_any(args, q, k, v, a, b, gk, h0, want_ht, grad && !env_is_1("HDLA_RECOMPUTE"));
        if (grad) {
            node = make_node<ChunkNode>();
            node->args = args;
            node->q.save(q); node->k.save(k); node->v.save(v); node->a.save(a); node->b.save(b); node->gk.save(gk);
            node->h0.save(h0);
            node->ws = r.ws;
            node->force_simt = r.forced_simt;
            node->a_type = a_.scalar_type();
            node->h0_type = h0_.defined() ? h0_.scalar_type() : at::kFloat;
        }
    }
    if (grad) {
        node->set_next_edges(torch::autograd::collect_next_edges(q_, k_, v_, a_, b_, gk_, h0_));
        torch::autograd::create_gradient_edge(r.o, node);
        if (r.ht.defined()) torch::autograd::create_gradient_edge(r.ht, node);
    }
    return {r.o, r.ht};
}

struct NormGateNode : torch::autograd::Node {
    Saved x, gate, w;
    double eps = 0;
    at::ScalarType gate_type, w_type;

    std::string name() const override { return "HdlaNormGateBackward"; }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        x.var.reset_data(); gate.var.reset_data(); w.var.reset_data();
    }
    variable_list apply(variable_list&& grads) override {
        std::lock_guard<std::mutex> lock(mutex_);
        at::NoGradGuard no_grad;
        if (!grads[0].defined()) return variable_list(3);
        const char* me = "HdlaNormGateBackward";
        const Tensor xs = x.get(me), gs = gate.get(me), ws = w.get(me);
        c10::cuda::CUDAGuard guard(xs.device());
        const Tensor d_o = grads[0].to(xs.scalar_type()).contiguous();
        Tensor dx = dense_like(xs), dg = dense_like(gs);
        const int64_t D = xs.size(-1);
        const cudaStream_t st = c10::cuda::getCurrentCUDAStream(xs.get_device()).stream();
        Tensor dw = dense({D}, at::kFloat, xs.device());
        check_cuda(cudaMemsetAsync(mptr(dw), 0, static_cast<size_t>(D) * 4, st), "dweight");
        check(abi.norm_gate_bwd(ptr(xs), ptr(gs), ptr(ws), ptr(d_o), mptr(dx), mptr(dg), fptr(dw), xs.numel() / D,
                                static_cast<int>(D), static_cast<float>(eps), dtype_code(xs), st), "hdla_norm_gate_bwd");
        return {dx, dg.to(gate_type), dw.to(w_type)};
    }
};

Tensor norm_gate_op(const Tensor& x_, const Tensor& gate_, const Tensor& w_, double eps) {
    const bool grad = needs_grad({&x_, &gate_, &w_});
    Tensor o;
    std::shared_ptr<NormGateNode> node;
    {
        at::NoGradGuard no_grad;
        c10::cuda::CUDAGuard guard(x_.device());
        const Tensor x = x_.contiguous(), gate = gate_.to(x.scalar_type()).contiguous(), w = w_.to(x.scalar_type()).contiguous();
        const int64_t D = x.size(-1);
        o = dense_like(x);
        check(abi.norm_gate_fwd(ptr(x), ptr(gate), ptr(w), mptr(o), x.numel() / D, static_cast<int>(D),
                                static_cast<float>(eps), dtype_code(x),
                                c10::cuda::getCurrentCUDAStream(x.get_device()).stream()), "hdla_norm_gate_fwd");
        if (grad) {
            node = make_node<NormGateNode>();
            node->x.save(x); node->gate.save(gate); node->w.save(w);
            node->eps = eps; node->gate_type = gate_.scalar_type(); node->w_type = w_.scalar_type();
        }
    }
    if (grad) {
        node->set_next_edges(torch::autograd::collect_next_edges(x_, gate_, w_));
        torch::autograd::create_gradient_edge(o, node);
    }
    return o;
}

// ------------------------------------------------------------------------------------------ Python functions
// Runs f without the GIL and turns C++ exceptions into Python ones as PyTorch's own bindings do: a Python exception
// that travelled through C++ (raised by a saved-tensor hook, say: non-reentrant checkpointing ends its recomputation
// with one) arrives as itself, an allocator's as torch.OutOfMemoryError.  False if an exception is set.
template <typename F>
bool guarded(F f) {
    std::exception_ptr err;
    bool python = false;
    PyThreadState* ts = PyEval_SaveThread();
    try {
        f();
    } catch (const PythonError&) {
        python = true;
    } catch (...) {
        err = std::current_exception();
    }
    PyEval_RestoreThread(ts);
    if (err) torch::translate_exception_to_python(err);
    return !err && !python;
}

// A tensor argument of the ordinary case, or null; None is an undefined tensor where `optional`.
const Tensor kNone;
const Tensor* arg(PyObject* o, bool optional = false) {
    if (o == Py_None) return optional ? &kNone : nullptr;
    const Tensor* t = as_tensor(o);
    if (!t || !t->is_cuda() || t->layout() != at::kStrided || t->_fw_grad(0).defined()) return nullptr;
    return t;
}
bool same_device(const Tensor& q, std::initializer_list<const Tensor*> ts) {
    for (const Tensor* t : ts)
        if (t->defined() && t->device() != q.device()) return false;
    return true;
}
bool shape_is(const Tensor& t, int64_t a, int64_t b, int64_t c, int64_t d) {
    return t.dim() == 4 && t.size(0) == a && t.size(1) == b && t.size(2) == c && t.size(3) == d;
}
bool fits_int(std::initializer_list<int64_t> v) {
    for (int64_t x : v)
        if (x <= 0 || x > 0x7fffffff) return false;
    return true;
}
#define NOT_MINE() do { Py_INCREF(Py_NotImplemented); return Py_NotImplemented; } while (0)

// offsets of a packed batch: a tuple of ints rising from 0 to T
bool offsets_arg(PyObject* o, int64_t T, std::vector<int64_t>& cu) {
    if (o == Py_None) return true;
    if (!PyTuple_Check(o) || PyTuple_GET_SIZE(o) < 2) return false;
    const Py_ssize_t n = PyTuple_GET_SIZE(o);
    cu.resize(n);
    for (Py_ssize_t i = 0; i < n; ++i) {
        cu[i] = PyLong_AsLongLong(PyTuple_GET_ITEM(o, i));
        if (cu[i] == -1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
        if (i == 0 ? cu[0] != 0 : cu[i] < cu[i - 1]) return false;
    }
    return cu.back() == T;
}

struct ChunkCall {
    const Tensor *q, *k, *v, *a, *b, *gk, *h0;
    ChunkArgs c;
};
// The arguments (q, k, v, a, b, gk, rank, scale or None, h0 or None) at av and chunk size and offsets; false: not the
// ordinary case.  With b None, a is beta (the layer's parametrisation inside the operator) and `rank` holds flag bits.
bool chunk_call(PyObject* const* av, PyObject* chunk, PyObject* offsets, ChunkCall& x) {
    const bool param_ab = av[4] == Py_None;
    const Tensor *q = x.q = arg(av[0]), *k = x.k = arg(av[1]), *v = x.v = arg(av[2]), *a = x.a = arg(av[3]),
                 *b = x.b = arg(av[4], true), *gk = x.gk = arg(av[5]), *h0 = x.h0 = arg(av[8], true);
    if (!abi.chunk_fwd || !q || !k || !v || !a || !b || !gk || !h0 || transforms_active()) return false;
    if (q->dim() != 4 || v->dim() != 4) return false;
    const int64_t B = q->size(0), T = q->size(1), H = q->size(2), K = q->size(3), V = v->size(3);
    int64_t R = PyLong_AsLongLong(av[6]), C = PyLong_AsLongLong(chunk);
    double scale = av[7] == Py_None ? 1.0 / std::sqrt(static_cast<double>(K)) : PyFloat_AsDouble(av[7]);
    if (PyErr_Occurred()) { PyErr_Clear(); return false; }
    int flags = 0;
    if (param_ab) { flags = static_cast<int>(R) | HDLA_FLAG_PARAM_AB; R = 2; }
    if (!same_device(*q, {k, v, a, b, gk, h0}) || dtype_code(*q) < 0 || dtype_code(*gk) < 0 ||
        k->scalar_type() != q->scalar_type() || v->scalar_type() != q->scalar_type() || !fits_int({B, T, H, K, V, R, C}))
        return false;
    if (!shape_is(*k, B, T, H, K) || !shape_is(*gk, B, T, H, K) || !shape_is(*v, B, T, H, V)) return false;
    if (param_ab) {
        if (a->numel() != B * T * H || a->dim() < 3 || a->size(0) != B || a->size(1) != T || a->size(2) != H ||
            !a->is_floating_point())
            return false;
    } else if (!shape_is(*a, B, T * R, H, K) || !shape_is(*b, B, T * R, H, K) || a->scalar_type() != q->scalar_type() ||
               b->scalar_type() != q->scalar_type()) {
        return false;
    }
    ChunkArgs& c = x.c;
    if (!offsets_arg(offsets, T, c.cu)) return false;
    c.n_states = static_cast<int>(c.cu.empty() ? B : static_cast<int64_t>(c.cu.size()) - 1);
    if (h0->defined() && !(shape_is(*h0, c.n_states, H, K, V) && h0->is_floating_point())) return false;
    const bool simt = env_is_1("HDLA_FORCE_SIMT"), honor = env_is_1("HDLA_HONOR_CHUNK"), tc = tc_shape(*q, T, K, V, R);
    if ((param_ab || !c.cu.empty()) && (!tc || simt || honor || (!c.cu.empty() && B != 1))) return false;
    // The result does not depend on the chunk size: what the tensor-core pipeline takes runs at its chunk of 64.
    if (tc && !simt && !honor) C = 64;
    if (simt) flags |= HDLA_FLAG_FORCE_SIMT;
    if (env_is_1("HDLA_FUSED_PREP")) flags |= HDLA_FLAG_FUSED_PREP;
    c.d.B = (int)B; c.d.T = (int)T; c.d.H = (int)H; c.d.K = (int)K; c.d.V = (int)V; c.d.R = (int)R; c.d.C = (int)C;
    c.d.dtype = dtype_code(*q); c.d.gk_dtype = dtype_code(*gk); c.d.flags = flags;
    c.scale = scale;
    return true;
}

PyObject* tuple_of(std::initializer_list<const Tensor*> ts) {
    PyObject* out = PyTuple_New(static_cast<Py_ssize_t>(ts.size()));
    Py_ssize_t i = 0;
    for (const Tensor* t : ts) PyTuple_SET_ITEM(out, i++, wrap(*t));
    return out;
}

// chunk(q, k, v, a, b, gk, rank, scale or None, h0 or None, output_final_state, chunk_size, offsets or None, keep or None)
//   keep None: the differentiable operator, (o, final state); None where the parametrisation's decay overflows (the
//   caller takes its two-call route).  keep True / False: a bare forward call, (o, final state, workspace kept for the
//   backward call or None, whether it ran on the fp32 pipeline)
PyObject* py_chunk(PyObject*, PyObject* const* av, Py_ssize_t n) {
    if (n != 13) { PyErr_SetString(PyExc_TypeError, "chunk takes 13 arguments"); return nullptr; }
    ChunkCall x;
    const bool bare = av[12] != Py_None, keep = av[12] == Py_True;
    const int want_ht = PyObject_IsTrue(av[9]);
    if (want_ht < 0) { PyErr_Clear(); NOT_MINE(); }
    if ((!bare && tracing()) || !chunk_call(av, av[10], av[11], x)) NOT_MINE();
    ChunkOut r;
    bool overflow = false;
    if (!guarded([&] {
            try {
                if (bare) {
                    at::NoGradGuard no_grad;
                    r = chunk_forward_any(x.c, x.q->contiguous(), x.k->contiguous(), x.v->contiguous(), x.a->contiguous(),
                                          x.b->defined() ? x.b->contiguous() : *x.b, x.gk->contiguous(),
                                          f32_contiguous(*x.h0), want_ht, keep);
                } else {
                    std::tie(r.o, r.ht) = chunk_op(x.c, *x.q, *x.k, *x.v, *x.a, *x.b, *x.gk, *x.h0, want_ht);
                }
            } catch (const DecayOverflow&) {
                overflow = true;
            }
        }))
        return nullptr;
    if (overflow) Py_RETURN_NONE;
    if (!bare) return tuple_of({&r.o, &r.ht});
    PyObject* out = PyTuple_New(4);
    PyTuple_SET_ITEM(out, 0, wrap(r.o));
    PyTuple_SET_ITEM(out, 1, wrap(r.ht));
    PyTuple_SET_ITEM(out, 2, wrap(r.ws));
    PyTuple_SET_ITEM(out, 3, PyBool_FromLong(r.forced_simt));
    return out;
}

// chunk_backward(q, k, v, a, b, gk, rank, scale, h0 or None, do, dht or None, workspace or None, chunk_size, offsets or
// None, forward ran on the fp32 pipeline) -> (dq, dk, dv, da, db, dgk, dh0 or None)
PyObject* py_chunk_backward(PyObject*, PyObject* const* av, Py_ssize_t n) {
    if (n != 15) { PyErr_SetString(PyExc_TypeError, "chunk_backward takes 15 arguments"); return nullptr; }
    ChunkCall x;
    const Tensor *d_o = arg(av[9], true), *dht = arg(av[10], true), *ws = arg(av[11], true);
    const bool simt = av[14] == Py_True;
    if (!chunk_call(av, av[12], av[13], x) || !d_o || !dht || !ws) {
        PyErr_SetString(PyExc_TypeError, "chunk_backward: arguments of another kind than the forward call's");
        return nullptr;
    }
    ChunkGrads g;
    if (!guarded([&] {
            at::NoGradGuard no_grad;
            g = chunk_backward(x.c, x.q->contiguous(), x.k->contiguous(), x.v->contiguous(), x.a->contiguous(),
                               x.b->defined() ? x.b->contiguous() : *x.b, x.gk->contiguous(), f32_contiguous(*x.h0), *d_o,
                               *dht, *ws, simt);
        }))
        return nullptr;
    return tuple_of({&g.dq, &g.dk, &g.dv, &g.da, &g.db, &g.dgk, &g.dh0});
}

// recurrent(q, k, v, a, b, gk, rank, scale or None, h0 or None, output_final_state, reverse, cu_seqlens or None)
PyObject* py_recurrent(PyObject*, PyObject* const* av, Py_ssize_t n) {
    if (n != 12) { PyErr_SetString(PyExc_TypeError, "recurrent takes 12 arguments"); return nullptr; }
    const Tensor *q = arg(av[0]), *k = arg(av[1]), *v = arg(av[2]), *a = arg(av[3]), *b = arg(av[4]), *gk = arg(av[5]),
                 *h0 = arg(av[8], true), *cu = arg(av[11], true);
    if (!abi.recurrent_fwd || !q || !k || !v || !a || !b || !gk || !h0 || !cu || transforms_active() || tracing()) NOT_MINE();
    if (needs_grad({q, k, v, a, b, gk, h0}) || q->dim() != 4 || v->dim() != 4) NOT_MINE();
    const int64_t B = q->size(0), T = q->size(1), H = q->size(2), K = q->size(3), V = v->size(3);
    const int64_t R = PyLong_AsLongLong(av[6]);
    const double scale = av[7] == Py_None ? 1.0 / std::sqrt(static_cast<double>(K)) : PyFloat_AsDouble(av[7]);
    const int want_ht = PyObject_IsTrue(av[9]), reverse = PyObject_IsTrue(av[10]);
    if (PyErr_Occurred()) { PyErr_Clear(); NOT_MINE(); }
    const auto dt = q->scalar_type();
    if (!same_device(*q, {k, v, a, b, gk, h0, cu}) || dtype_code(*q) < 0 || dtype_code(*gk) < 0 || k->scalar_type() != dt ||
        v->scalar_type() != dt || a->scalar_type() != dt || b->scalar_type() != dt || !fits_int({B, T, H, K, V, R}))
        NOT_MINE();
    if (!shape_is(*k, B, T, H, K) || !shape_is(*gk, B, T, H, K) || !shape_is(*v, B, T, H, V) ||
        !shape_is(*a, B, T * R, H, K) || !shape_is(*b, B, T * R, H, K))
        NOT_MINE();
    int64_t N = B;
    if (cu->defined()) {
        if (B != 1 || cu->dim() != 1 || cu->size(0) < 2 || cu->is_floating_point()) NOT_MINE();
        N = cu->size(0) - 1;
    }
    if (h0->defined() && !(shape_is(*h0, N, H, K, V) && h0->is_floating_point())) NOT_MINE();
    HdlaDims d{};
    d.B = (int)B; d.T = (int)T; d.H = (int)H; d.K = (int)K; d.V = (int)V; d.R = (int)R;
    d.dtype = dtype_code(*q); d.gk_dtype = dtype_code(*gk);
    Tensor o, ht;
    if (!guarded([&] {
            at::NoGradGuard no_grad;
            c10::cuda::CUDAGuard guard(q->device());
            const Tensor qc = q->contiguous(), kc = k->contiguous(), vc = v->contiguous(), ac = a->contiguous(),
                         bc = b->contiguous(), gc = gk->contiguous(), hc = f32_contiguous(*h0),
                         cc = cu->defined() ? cu->to(at::kLong).contiguous() : *cu;
            o = dense_like(vc);
            if (want_ht) ht = dense({N, H, K, V}, at::kFloat, qc.device());
            check(abi.recurrent_fwd(&d, ptr(qc), ptr(kc), ptr(vc), ptr(ac), ptr(bc), ptr(gc), static_cast<float>(scale),
                                    fptr(hc), mptr(o), fptr(ht), static_cast<const int64_t*>(ptr(cc)), (int)N, reverse,
                                    c10::cuda::getCurrentCUDAStream(qc.get_device()).stream()), "hdla_recurrent_fwd");
        }))
        return nullptr;
    return tuple_of({&o, &ht});
}

// norm_gate(x, gate, weight, eps)
PyObject* py_norm_gate(PyObject*, PyObject* const* av, Py_ssize_t n) {
    if (n != 4) { PyErr_SetString(PyExc_TypeError, "norm_gate takes 4 arguments"); return nullptr; }
    const Tensor *x = arg(av[0]), *gate = arg(av[1]), *w = arg(av[2]);
    if (!abi.norm_gate_fwd || !x || !gate || !w || transforms_active() || tracing()) NOT_MINE();
    const double eps = PyFloat_AsDouble(av[3]);
    if (PyErr_Occurred()) { PyErr_Clear(); NOT_MINE(); }
    if (dtype_code(*x) < 0 || x->dim() < 1 || x->numel() == 0 || gate->sizes() != x->sizes() || w->dim() != 1 ||
        w->size(0) != x->size(-1) || !same_device(*x, {gate, w}) || !gate->is_floating_point() || !w->is_floating_point())
        NOT_MINE();
    Tensor o;
    if (!guarded([&] { o = norm_gate_op(*x, *gate, *w, eps); })) return nullptr;
    return wrap(o);
}

// status functions: check(dev index or -1, wait), post(workspace tensor), decay(dev), set_decay(dev, x or None)
PyObject* py_status_check(PyObject*, PyObject* const* av, Py_ssize_t n) {
    if (n != 2) { PyErr_SetString(PyExc_TypeError, "status_check(device index or -1, wait)"); return nullptr; }
    const long dev = PyLong_AsLong(av[0]);
    const int wait = PyObject_IsTrue(av[1]);
    if (PyErr_Occurred()) return nullptr;
    if (!guarded([&] {
            std::vector<int> devs;
            {
                Lock lk(g_mu);
                for (auto& e : g_devices)
                    if (dev < 0 || e.first == dev) devs.push_back(e.first);
            }
            for (int i : devs) status_check(i, wait != 0);
        }))
        return nullptr;
    Py_RETURN_NONE;
}
PyObject* py_status_post(PyObject*, PyObject* ws) {
    const Tensor* t = arg(ws);
    if (!t || t->nbytes() < 16) { PyErr_SetString(PyExc_TypeError, "status_post takes a CUDA workspace"); return nullptr; }
    if (!guarded([&] {
            c10::cuda::CUDAGuard guard(t->device());
            const cudaStream_t st = c10::cuda::getCurrentCUDAStream(t->get_device()).stream();
            status_post(ptr(*t), t->get_device(), st, capturing(st));
        }))
        return nullptr;
    Py_RETURN_NONE;
}
PyObject* py_decay(PyObject*, PyObject* dev) {
    const long i = PyLong_AsLong(dev);
    if (PyErr_Occurred()) return nullptr;
    double x = NAN;
    if (!guarded([&] { x = board_of((int)i).decay(); })) return nullptr;
    if (x != x) Py_RETURN_NONE;
    return PyFloat_FromDouble(x);
}
PyObject* py_set_decay(PyObject*, PyObject* const* av, Py_ssize_t n) {
    if (n != 2) { PyErr_SetString(PyExc_TypeError, "set_decay(device index, value or None)"); return nullptr; }
    const long i = PyLong_AsLong(av[0]);
    const double x = av[1] == Py_None ? NAN : PyFloat_AsDouble(av[1]);
    if (PyErr_Occurred()) return nullptr;
    if (!guarded([&] { board_of((int)i).set_decay(x); })) return nullptr;
    Py_RETURN_NONE;
}

// bind(handle of the loaded libhdla, callable that warns of the fp32 rerun)
PyObject* py_bind(PyObject*, PyObject* const* av, Py_ssize_t n) {
    if (n != 2) { PyErr_SetString(PyExc_TypeError, "bind(handle, on_overflow)"); return nullptr; }
    void* h = PyLong_AsVoidPtr(av[0]);
    if (PyErr_Occurred()) return nullptr;
    if (!guarded([&] {
            decltype(&hdla_version) version;
            look_up(h, "hdla_version", version);
            if (version() != HDLA_VERSION)
                throw std::runtime_error("_binding.so is built for version " + std::to_string(HDLA_VERSION) +
                                         " of libhdla, this is version " + std::to_string(version()));
            look_up(h, "hdla_chunk_workspace_bytes", abi.workspace_bytes);
            look_up(h, "hdla_chunk_uses_tensor_cores", abi.uses_tensor_cores);
            look_up(h, "hdla_fp32_status_words", abi.fp32_status_words);
            look_up(h, "hdla_chunk_bwd", abi.chunk_bwd);
            look_up(h, "hdla_norm_gate_fwd", abi.norm_gate_fwd);
            look_up(h, "hdla_norm_gate_bwd", abi.norm_gate_bwd);
            look_up(h, "hdla_last_error", abi.last_error);
            look_up(h, "hdla_recurrent_fwd", abi.recurrent_fwd);
            look_up(h, "hdla_chunk_fwd", abi.chunk_fwd);
        }))
        return nullptr;
    Py_XDECREF(g_on_overflow);
    Py_INCREF(av[1]);
    g_on_overflow = av[1];
    Py_RETURN_NONE;
}

// read from the file before it is loaded (build.py)
__attribute__((used)) const char kBuiltFor[] = HDLA_BUILT_FOR;

#define FAST(f) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL
PyMethodDef methods[] = {{"bind", FAST(py_bind), nullptr},
                         {"chunk", FAST(py_chunk), nullptr},
                         {"chunk_backward", FAST(py_chunk_backward), nullptr},
                         {"recurrent", FAST(py_recurrent), nullptr},
                         {"norm_gate", FAST(py_norm_gate), nullptr},
                         {"status_check", FAST(py_status_check), nullptr},
                         {"status_post", py_status_post, METH_O, nullptr},
                         {"decay", py_decay, METH_O, nullptr},
                         {"set_decay", FAST(py_set_decay), nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_binding", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__binding() { return PyModule_Create(&module); }
