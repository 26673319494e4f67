// Native host path of the package: argument checks, memory, autograd and kernel launches for the calls whose
// host time is a visible part of the whole (a decoding step runs for 4 us on the device, a short prefill for 50).
// The Python modules keep the public signatures and everything that is not on such a path.
//
// No tensor is kept from one call for the next; the only state here is the table of the devices' status words.
#include <ATen/MemoryOverlap.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/extension.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <optional>
#include <string>

#include "../../include/kda_b200.h"

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

namespace {

constexpr int CHUNK = KDA_CHUNK;

// ---- per-device status word and its pinned host mirror (owned by ops._DeviceStatus) -------------------------
constexpr int MAX_DEVICES = 64;
struct StatusWord {
    std::atomic<int32_t*> dev{nullptr};  // set after host: calls of other threads look without the interpreter lock
    const volatile int32_t* host = nullptr;
};
StatusWord g_status[MAX_DEVICES];
// Python callables: status_of(device_index) creates the words; report(device_index) raises and clears;
// guard_span() reads the mutable span of the guard contract
py::object* g_status_of = nullptr;
py::object* g_report = nullptr;
py::object* g_guard_span = nullptr;

void set_status(int device, int64_t dev_ptr, int64_t host_ptr) {
    TORCH_CHECK(device >= 0 && device < MAX_DEVICES, "device index out of range");
    g_status[device].host = reinterpret_cast<const volatile int32_t*>(host_ptr);
    g_status[device].dev.store(reinterpret_cast<int32_t*>(dev_ptr), std::memory_order_release);
}

void set_callbacks(py::object status_of, py::object report, py::object guard_span) {
    g_status_of = new py::object(std::move(status_of));  // (never destroyed: they outlive the interpreter's modules)
    g_report = new py::object(std::move(report));
    g_guard_span = new py::object(std::move(guard_span));
}

const StatusWord& status_word(int device) {
    TORCH_CHECK(device >= 0 && device < MAX_DEVICES, "device index out of range");
    const StatusWord& st = g_status[device];
    if (!st.dev.load(std::memory_order_acquire) || *st.host) {
        py::gil_scoped_acquire gil;
        if (!st.dev.load(std::memory_order_relaxed)) (*g_status_of)(device);
        if (*st.host) (*g_report)(device);  // a wait that gave up in an earlier call surfaces here
    }
    return st;
}

// the guard contract's span is a module attribute that callers may change between calls; it is read at every call
float guard_span() {
    py::gil_scoped_acquire gil;
    return (*g_guard_span)().cast<float>();
}

// debugging / A-B switches of the environment (ops.chunk_kda documents them), read at every call
int64_t env_flags() {
    auto is_one = [](const char* n) { const char* v = std::getenv(n); return v && v[0] == '1' && !v[1]; };
    int64_t f = 0;
    if (is_one("OPENKIMI_B200_FP32_MATH")) f |= KDA_FLAG_FORCE_SIMT;
    if (is_one("OPENKIMI_B200_ROW_COPIES")) f |= KDA_FLAG_ROW_COPIES;
    if (const char* v = std::getenv("OPENKIMI_B200_FP32_STAGES")) f |= (std::strtol(v, nullptr, 10) & 31) << 5;
    return f;
}

void check_rc(int rc, const char* what) {
    if (rc == KDA_OK) return;
    std::string msg = std::string(what) + " failed: " + kda_status_string(rc);
    const std::string extra = kda_last_cuda_error();
    if (rc == KDA_ERR_LAUNCH && !extra.empty()) msg += " (" + extra + ")";
    throw std::runtime_error(msg);
}

std::string shape_of(const Tensor& t) {
    std::string s = "(";
    for (int64_t i = 0; i < t.dim(); ++i) s += (i ? ", " : "") + std::to_string(t.size(i));
    return s + (t.dim() == 1 ? ",)" : ")");
}
[[noreturn]] void value_error(const std::string& m) { throw py::value_error(m); }
[[noreturn]] void type_error(const std::string& m) { throw py::type_error(m); }

void require_cuda(const Tensor& t) {
    if (!t.is_cuda()) throw std::runtime_error("chunk_kda runs only on a CUDA device (sm_100a); there is no CPU fallback");
}

// the kernels follow raw pointers: every tensor of a call has to be where q is
void require_device(const Tensor& q, const char* name, const Tensor& t) {
    if (t.defined() && t.device() != q.device())
        throw std::runtime_error(std::string("expected ") + name + " on " + q.device().str() + ", the device of q, but it is on " +
                                 t.device().str());
}

// A call that nobody differentiates backward does not pass through its autograd node, which refuses forward-mode inputs.
template <class Tensors>
void refuse_tangents(const Tensors& inputs) {
    for (const Tensor* t : inputs)
        if (t->defined() && t->_fw_grad(0).defined())
            throw std::runtime_error("the KDA kernels have no forward-mode derivative (an input carries a tangent)");
}

int dtype_code(const Tensor& t) {
    if (t.scalar_type() == at::kBFloat16) return KDA_DTYPE_BF16;
    if (t.scalar_type() == at::kFloat) return KDA_DTYPE_F32;
    type_error(std::string("q/k/v must be float32 or bfloat16, got ") + c10::toString(t.scalar_type()));
}

// contiguous, in dtype dt, starting on a 16-byte boundary (a view into the middle of a buffer is copied)
Tensor ready(const Tensor& t, at::ScalarType dt) {
    Tensor r = t.scalar_type() == dt ? t : t.to(dt);
    if (!r.is_contiguous()) r = r.contiguous();
    return (reinterpret_cast<uintptr_t>(r.data_ptr()) & 15) == 0 ? r : r.clone();
}
// the same without a new reference where t is that already or undefined; copy holds what else it becomes
const Tensor& ready(const Tensor& t, at::ScalarType dt, Tensor& copy) {
    if (!t.defined() || (t.scalar_type() == dt && t.is_contiguous() && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0)) return t;
    return copy = ready(t, dt);
}
// a new tensor without the dispatcher's detour (half of what at::empty costs)
Tensor fresh(at::IntArrayRef sizes, at::ScalarType dt, const Tensor& like) {
    return Tensor(at::detail::empty_cuda(sizes, dt, like.device(), std::nullopt));
}
const Tensor& val(const OptTensor& t) {
    static const Tensor none;
    return t ? *t : none;
}
template <class T>
T* ptr(const Tensor& t) { return t.defined() ? static_cast<T*>(t.data_ptr()) : nullptr; }

void* stream_of(const Tensor& t) { return at::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// ---- recurrent steps -----------------------------------------------------------------------------------------
// q, k, g, v: [N, (T,) H, K]; multi says whether the token axis is there
std::tuple<Tensor, OptTensor> recurrent(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta,
                                        const OptTensor& state, const OptTensor& A_log, const OptTensor& dt_bias,
                                        std::optional<double> scale, bool l2norm, bool gate, bool sigmoid, bool v_first,
                                        bool inplace, bool multi, bool want_state) {
    require_cuda(q);
    const Tensor &a0 = gate ? val(A_log) : val(std::nullopt), &b0 = gate ? val(dt_bias) : val(std::nullopt), &s0 = val(state);
    require_device(q, "k", k); require_device(q, "v", v); require_device(q, "g", g); require_device(q, "beta", beta);
    require_device(q, "state", s0); require_device(q, "A_log", a0); require_device(q, "dt_bias", b0);
    const int64_t dims = multi ? 4 : 3;
    if (q.dim() != dims || q.sizes() != k.sizes() || g.sizes() != q.sizes())
        value_error("q, k, g must share one shape " + std::string(multi ? "[B,T,H,K]" : "[N,H,K]") + ", got " + shape_of(q) + ", " +
                    shape_of(k) + ", " + shape_of(g));
    const int64_t N = q.size(0), T = multi ? q.size(1) : 1, H = q.size(dims - 2), K = q.size(dims - 1);
    if (v.sizes() != q.sizes() || (K != 64 && K != 128))
        value_error("the B200 KDA kernels need K == V in (64, 128), got K=" + std::to_string(K) + ", v=" + shape_of(v));
    if (beta.sizes() != q.sizes().slice(0, dims - 1))
        value_error("beta must have the shape of q without its last axis, got " + shape_of(beta));
    const int dtype = dtype_code(q);
    const std::array<int64_t, 4> want = {N, H, K, K};
    if (!state && !multi) type_error("recurrent_kda_step needs a state");
    if (state && (state->scalar_type() != at::kFloat || state->sizes() != at::IntArrayRef(want)))
        value_error("state must be float32 [N,H," + std::to_string(K) + "," + std::to_string(K) + "], got " +
                    c10::toString(state->scalar_type()) + " " + shape_of(*state));
    if (gate && (!A_log || A_log->numel() != H || (dt_bias && dt_bias->numel() != H * K)))
        value_error("use_gate_in_kernel=True needs A_log with H entries (and dt_bias with H*K entries)");
    at::NoGradGuard no_grad;
    c10::cuda::CUDAGuard guard(q.device());
    const auto dt = q.scalar_type();
    Tensor copies[8];
    const Tensor &qc = ready(q, dt, copies[0]), &kc = ready(k, dt, copies[1]), &vc = ready(v, dt, copies[2]),
                 &gc = ready(g, dt, copies[3]), &bc = ready(beta, dt, copies[4]), &a = ready(a0, at::kFloat, copies[5]),
                 &b = ready(b0, at::kFloat, copies[6]), &s_in = ready(s0, at::kFloat, copies[7]);
    Tensor s_out, s_back;  // s_back: a state to be updated that the kernel cannot write itself
    if (want_state) {
        const Tensor own = inplace ? (state->requires_grad() ? state->detach() : *state) : Tensor();
        if (inplace && s_in.data_ptr() == own.data_ptr()) {
            s_out = own;
        } else {
            s_out = fresh(want, at::kFloat, q);
            // (an expanded state has no memory of its own to update: the new state is returned alone)
            if (inplace && at::has_internal_overlap(own) != at::MemOverlap::Yes) s_back = own;
        }
    }
    Tensor o = fresh(q.sizes(), dt, q);
    status_word(q.device().index());
    if (N * T * H == 0) {
        if (s_out.defined() && !s_out.is_same(s_in)) {
            if (s_in.defined()) s_out.copy_(s_in);
            else s_out.zero_();
        }
        return {o, want_state ? OptTensor(s_out) : OptTensor()};
    }
    const int flags = (l2norm ? KDA_FLAG_QK_L2NORM : 0) | (gate ? KDA_FLAG_GATE : 0) | (sigmoid ? KDA_FLAG_BETA_SIGMOID : 0) |
                      (v_first ? KDA_FLAG_STATE_V_FIRST : 0);
    check_rc(kda_recurrent_fwd(qc.data_ptr(), kc.data_ptr(), vc.data_ptr(), gc.data_ptr(), bc.data_ptr(), ptr<float>(a), ptr<float>(b),
                               ptr<float>(s_in), ptr<float>(s_out), o.data_ptr(), (int)N, (int)T, (int)H, (int)K, (int)K, dtype, flags,
                               (float)scale.value_or(1.0 / std::sqrt((double)K)), stream_of(q)),
             "kda_recurrent_fwd");
    if (s_back.defined()) s_out = s_back.copy_(s_out);
    return {o, want_state ? OptTensor(s_out) : OptTensor()};
}

// ---- chunk_kda -----------------------------------------------------------------------------------------------
// what forward and backward of one call share besides the tensors
struct Spec {
    double scale = 1.0;
    int flags = 0;
    bool output_final_state = false, keep = false;
    int64_t NT = 0;       // chunks over all sequences
    int64_t longest = 0;  // chunks of the longest packed document
};
struct Inputs {
    Tensor q, k, v, g, beta, A_log, dt_bias, h0, conv_q, conv_k, conv_v;  // contiguous; undefined where absent
    Tensor cu, chunk_seq, seq_off, chunk_tab;                             // packed documents only
};

struct Prepared {
    KdaParams p{};
    size_t fwd_bytes = 0, bwd_bytes = 0;
    int64_t N = 0;
    bool empty = false;
};

Prepared prepare(const Inputs& in, const Spec& sp, int flags) {
    Prepared r;
    KdaParams& p = r.p;
    const Tensor& q = in.q;
    p.B = (int)q.size(0); p.T = (int)q.size(1); p.H = (int)q.size(2); p.dk = (int)q.size(3); p.dv = (int)in.v.size(3);
    r.N = in.cu.defined() ? in.cu.numel() - 1 : q.size(0);
    r.empty = sp.NT == 0;
    p.N = (int)r.N;
    p.max_chunks = (int)sp.longest;
    p.NT = (int)std::max<int64_t>(sp.NT, 1);
    p.dtype = q.scalar_type() == at::kBFloat16 ? KDA_DTYPE_BF16 : KDA_DTYPE_F32;
    p.flags = flags;
    p.scale = (float)sp.scale;
    p.guard_span = guard_span();
    p.q = q.data_ptr(); p.k = in.k.data_ptr(); p.v = in.v.data_ptr(); p.g = in.g.data_ptr(); p.beta = in.beta.data_ptr();
    p.A_log = ptr<float>(in.A_log); p.dt_bias = ptr<float>(in.dt_bias); p.h0 = ptr<float>(in.h0);
    if (in.cu.defined()) {
        p.cu_seqlens = ptr<int64_t>(in.cu); p.chunk_seq = ptr<int32_t>(in.chunk_seq);
        p.seq_chunk_off = ptr<int32_t>(in.seq_off); p.chunk_tab = ptr<int32_t>(in.chunk_tab);
    }
    if (in.conv_q.defined()) {
        p.conv_q = ptr<float>(in.conv_q); p.conv_k = ptr<float>(in.conv_k); p.conv_v = ptr<float>(in.conv_v);
        p.conv_ksize = (int)in.conv_q.size(-1);
    }
    const StatusWord& st = status_word(q.device().index());
    p.status = st.dev.load(std::memory_order_relaxed);
    p.status_host = const_cast<int32_t*>(st.host);
    check_rc(kda_workspace_bytes(&p, &r.fwd_bytes, &r.bwd_bytes), "kda_workspace_bytes");
    return r;
}

Tensor bytes(size_t n, const Tensor& like) { return fresh({(int64_t)n}, at::kByte, like); }
Tensor fresh_like(const Tensor& t) { return fresh(t.sizes(), t.scalar_type(), t); }

std::array<int64_t, 4> state_shape(const Inputs& in, const Spec& sp, int64_t N) {
    const int64_t H = in.q.size(2), dk = in.q.size(3), dv = in.v.size(3);
    if (sp.flags & KDA_FLAG_STATE_V_FIRST) return {N, H, dv, dk};
    return {N, H, dk, dv};
}

struct FwdOut { Tensor o, ht, ws, borders; };

// recompute: the backward will rebuild the records; the states at the split points of long sequences are kept for it
FwdOut run_fwd(const Inputs& in, const Spec& sp, bool recompute = false) {
    // The forward-only kernels skip every record that only the backward reads: when nobody will differentiate this
    // call, or the backward rebuilds the records anyway (recompute policy).
    Prepared pr = prepare(in, sp, sp.keep ? sp.flags : sp.flags | KDA_FLAG_NO_SAVE);
    FwdOut out;
    const Tensor& q = in.q;
    if (recompute && !pr.empty) {
        size_t n = 0;
        check_rc(kda_border_bytes(&pr.p, &n), "kda_border_bytes");
        if (n) {
            out.borders = bytes(n, q);
            pr.p.borders = ptr<float>(out.borders);
            check_rc(kda_workspace_bytes(&pr.p, &pr.fwd_bytes, &pr.bwd_bytes), "kda_workspace_bytes");
        }
    }
    out.o = fresh_like(in.v);
    if (sp.output_final_state) out.ht = fresh(state_shape(in, sp, pr.N), at::kFloat, q);
    out.ws = bytes(pr.fwd_bytes, q);
    if (pr.empty) {
        if (out.ht.defined()) {
            if (in.h0.defined()) out.ht.copy_(in.h0);
            else out.ht.zero_();
        }
        return out;
    }
    pr.p.o = out.o.data_ptr(); pr.p.ht = ptr<float>(out.ht);
    pr.p.workspace = out.ws.data_ptr(); pr.p.workspace_bytes = pr.fwd_bytes;
    check_rc(kda_fwd(&pr.p, stream_of(q)), "kda_fwd");
    return out;
}

struct Grads { Tensor q, k, v, g, beta, A_log, dt_bias, h0, conv_q, conv_k, conv_v; };

// out: where dq, dk, dv, dg go if the caller has a place for them
Grads run_bwd(const Inputs& in, const Spec& sp, Tensor ws, const Tensor& borders, const Tensor& grad_o, const Tensor& grad_ht, Grads out = {}) {
    Prepared pr = prepare(in, sp, sp.flags);
    if (borders.defined()) {
        pr.p.borders = ptr<float>(borders);
        check_rc(kda_workspace_bytes(&pr.p, &pr.fwd_bytes, &pr.bwd_bytes), "kda_workspace_bytes");
    }
    const Tensor& q = in.q;
    const int64_t H = q.size(2), dk = q.size(3);
    void* stream = stream_of(q);
    KdaParams& p = pr.p;
    if (!ws.defined()) {  // recompute policy: rebuild the per-chunk records instead of keeping them
        ws = bytes(pr.fwd_bytes, q);
        p.o = q.data_ptr();  // (not written)
        p.workspace = ws.data_ptr(); p.workspace_bytes = pr.fwd_bytes;
        p.flags |= KDA_FLAG_NO_OUTPUT | (borders.defined() ? KDA_FLAG_BORDERS_READY : 0);
        if (!pr.empty) check_rc(kda_fwd(&p, stream), "kda_fwd (recompute)");
        p.flags = sp.flags;
    }
    const Tensor go = grad_o.defined() ? ready(grad_o, q.scalar_type()) : at::zeros_like(in.v);
    const Tensor ght = grad_ht.defined() ? ready(grad_ht, at::kFloat) : Tensor();
    if (!out.q.defined()) out.q = fresh_like(q);
    if (!out.k.defined()) out.k = fresh_like(in.k);
    if (!out.v.defined()) out.v = fresh_like(in.v);
    if (!out.g.defined()) out.g = fresh_like(in.g);
    if (!out.beta.defined()) out.beta = fresh_like(in.beta);
    const bool gate = sp.flags & KDA_FLAG_GATE;
    // written in full by the fixed-order reduction kernel (no zero fill needed)
    if (gate) out.A_log = fresh({H}, at::kFloat, q);
    if (gate && in.dt_bias.defined()) out.dt_bias = fresh({H * dk}, at::kFloat, q);
    if (in.h0.defined()) out.h0 = fresh(state_shape(in, sp, pr.N), at::kFloat, q);
    if (in.conv_q.defined()) {
        const std::array<int64_t, 2> sh = {H * dk, in.conv_q.size(-1)};
        out.conv_q = fresh(sh, at::kFloat, q); out.conv_k = fresh(sh, at::kFloat, q); out.conv_v = fresh(sh, at::kFloat, q);
    }
    if (pr.empty) {
        for (Tensor* t : {&out.q, &out.k, &out.v, &out.g, &out.beta, &out.A_log, &out.dt_bias, &out.conv_q, &out.conv_k, &out.conv_v})
            if (t->defined()) t->zero_();
        if (out.h0.defined()) {
            if (ght.defined()) out.h0.copy_(ght);
            else out.h0.zero_();
        }
        return out;
    }
    Tensor scratch = bytes(pr.bwd_bytes, q);
    p.o = out.q.data_ptr();  // unused by the backward; must be non-NULL
    p.ht = nullptr;
    p.workspace = ws.data_ptr(); p.workspace_bytes = pr.fwd_bytes;
    p.grad_o = go.data_ptr(); p.grad_ht = ptr<float>(ght);
    p.grad_q = out.q.data_ptr(); p.grad_k = out.k.data_ptr(); p.grad_v = out.v.data_ptr(); p.grad_g = out.g.data_ptr();
    p.grad_beta = out.beta.data_ptr();
    p.grad_A_log = ptr<float>(out.A_log); p.grad_dt_bias = ptr<float>(out.dt_bias); p.grad_h0 = ptr<float>(out.h0);
    p.grad_conv_q = ptr<float>(out.conv_q); p.grad_conv_k = ptr<float>(out.conv_k); p.grad_conv_v = ptr<float>(out.conv_v);
    p.bwd_scratch = scratch.data_ptr(); p.bwd_scratch_bytes = pr.bwd_bytes;
    check_rc(kda_bwd(&p, stream), "kda_bwd");
    return out;
}

Inputs gather(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, const Tensor& A_log,
              const Tensor& dt_bias, const Tensor& h0, const Tensor& cq, const Tensor& ck, const Tensor& cv, const Inputs& tables) {
    Inputs in = tables;
    const auto dt = q.scalar_type();
    in.q = ready(q, dt); in.k = ready(k, dt); in.v = ready(v, dt); in.g = ready(g, dt); in.beta = ready(beta, dt);
    if (A_log.defined()) in.A_log = ready(A_log, at::kFloat);
    if (dt_bias.defined()) in.dt_bias = ready(dt_bias, at::kFloat);
    if (h0.defined()) in.h0 = ready(h0, at::kFloat);
    if (cq.defined()) {  // filters [H*K, 1, ksize] -> [H*K, ksize]
        auto flat = [](const Tensor& w) { return ready(w.reshape({w.size(0), w.size(2)}), at::kFloat); };
        in.conv_q = flat(cq); in.conv_k = flat(ck); in.conv_v = flat(cv);
    }
    return in;
}

variable_list to_list(const Inputs& in, const Tensor& ws, const Tensor& borders) {
    return {in.q, in.k, in.v, in.g, in.beta, in.A_log, in.dt_bias, in.h0, in.conv_q, in.conv_k, in.conv_v,
            in.cu, in.chunk_seq, in.seq_off, in.chunk_tab, ws, borders};
}
Inputs from_list(const variable_list& s) {
    return {s[0], s[1], s[2], s[3], s[4], s[5], s[6], s[7], s[8], s[9], s[10], s[11], s[12], s[13], s[14]};
}
void save_spec(AutogradContext* ctx, const Spec& sp) {
    ctx->saved_data["scale"] = sp.scale;
    ctx->saved_data["flags"] = (int64_t)sp.flags;
    ctx->saved_data["NT"] = sp.NT;
    ctx->saved_data["longest"] = sp.longest;
    ctx->saved_data["keep"] = sp.keep;
}
Spec load_spec(AutogradContext* ctx) {
    Spec sp;
    sp.scale = ctx->saved_data["scale"].toDouble();
    sp.flags = (int)ctx->saved_data["flags"].toInt();
    sp.NT = ctx->saved_data["NT"].toInt();
    sp.longest = ctx->saved_data["longest"].toInt();
    sp.keep = ctx->saved_data["keep"].toBool();
    return sp;
}
Tensor as_filter(const Tensor& w) { return w.defined() ? w.view({w.size(0), 1, w.size(1)}) : w; }

OptTensor opt(const Tensor& t) { return t.defined() ? OptTensor(t) : OptTensor(); }  // (a node's inputs must be defined tensors)

struct ChunkKda : torch::autograd::Function<ChunkKda> {
    static variable_list forward(AutogradContext* ctx, Tensor q, Tensor k, Tensor v, Tensor g, Tensor beta, OptTensor A_log,
                                 OptTensor dt_bias, OptTensor h0, OptTensor cq, OptTensor ck, OptTensor cv, const Inputs& tables,
                                 const Spec& sp) {
        const Inputs in = gather(q, k, v, g, beta, val(A_log), val(dt_bias), val(h0), val(cq), val(ck), val(cv), tables);
        FwdOut f = run_fwd(in, sp, !sp.keep);
        ctx->save_for_backward(to_list(in, sp.keep ? f.ws : Tensor(), f.borders));
        ctx->set_materialize_grads(false);  // an unused final state has no gradient, rather than one of zeros
        save_spec(ctx, sp);
        if (f.ht.defined()) return {f.o, f.ht};
        return {f.o};
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const variable_list s = ctx->get_saved_variables();
        const Inputs in = from_list(s);
        c10::cuda::CUDAGuard guard(in.q.device());
        Grads r = run_bwd(in, load_spec(ctx), s[15], s[16], grads[0], grads.size() > 1 ? grads[1] : Tensor());
        // (the engine casts every gradient to its input's dtype)
        return {r.q, r.k, r.v, r.g, r.beta, r.A_log, r.dt_bias, r.h0, as_filter(r.conv_q), as_filter(r.conv_k), as_filter(r.conv_v),
                Tensor(), Tensor()};
    }
};

void take_tables(Inputs& tables, const OptTensor& cu, const OptTensor& chunk_seq, const OptTensor& seq_off, const OptTensor& chunk_tab,
                 int64_t batch) {
    if (batch != 1)
        value_error("The batch size is expected to be 1 rather than " + std::to_string(batch) +
                    " when using `cu_seqlens`.Please flatten variable-length inputs before processing.");
    tables.cu = *cu; tables.chunk_seq = *chunk_seq; tables.seq_off = *seq_off; tables.chunk_tab = *chunk_tab;
}

std::tuple<Tensor, OptTensor> chunk_kda(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta,
                                        OptTensor A_log, OptTensor dt_bias, OptTensor h0, OptTensor cq, OptTensor ck, OptTensor cv,
                                        std::optional<double> scale, int64_t flags, bool output_final_state, bool disable_recompute,
                                        OptTensor cu, OptTensor chunk_seq, OptTensor seq_off, OptTensor chunk_tab, int64_t NT, int64_t longest) {
    for (const Tensor* t : {&q, &k, &v, &g, &beta}) require_cuda(*t);
    if (q.dim() != 4 || q.sizes() != k.sizes())
        value_error("q and k must have the same shape [B,T,H,K], got q=" + shape_of(q) + " vs k=" + shape_of(k));
    const int64_t B = q.size(0), T = q.size(1), H = q.size(2), K = q.size(3);
    if (v.dim() != 4 || v.sizes().slice(0, 3) != q.sizes().slice(0, 3))
        value_error("grouped value heads (HV != H) are not supported: v must be [B,T,H,V]");
    if (g.sizes() != q.sizes()) value_error("g must have shape " + shape_of(q) + ", got " + shape_of(g));
    if (beta.sizes() != q.sizes().slice(0, 3)) value_error("beta must have shape [B,T,H] of q, got " + shape_of(beta));
    if (K != v.size(3) || (K != 64 && K != 128))
        value_error("the B200 KDA kernels need K == V in (64, 128), got K=" + std::to_string(K) + ", V=" + std::to_string(v.size(3)));
    dtype_code(q);
    Inputs tables;
    Spec sp;
    int64_t n_seq = B;
    if (cu) {
        n_seq = cu->numel() - 1;
        take_tables(tables, cu, chunk_seq, seq_off, chunk_tab, B);
        if (h0 && h0->size(0) != n_seq)
            value_error("The number of initial states is expected to be equal to the number of input sequences, i.e., " +
                        std::to_string(n_seq) + " rather than " + std::to_string(h0->size(0)) + ".");
        sp.NT = NT;
        sp.longest = longest;
    } else {
        sp.NT = B * ((T + CHUNK - 1) / CHUNK);
    }
    if (h0) {
        if (h0->scalar_type() != at::kFloat) type_error("initial_state must be in float32.");
        const std::array<int64_t, 4> want = {n_seq, H, K, K};
        if (h0->sizes() != at::IntArrayRef(want))
            value_error("initial_state must have shape (" + std::to_string(n_seq) + ", " + std::to_string(H) + ", " + std::to_string(K) +
                        ", " + std::to_string(K) + "), got " + shape_of(*h0));
    }
    Tensor a, b;
    if (flags & KDA_FLAG_GATE) {
        if (!A_log) value_error("A_log must be provided when use_gate_in_kernel=True.");
        if (A_log->numel() != H || (dt_bias && dt_bias->numel() != H * K))
            value_error("A_log must have H entries and dt_bias H*K entries");
        a = A_log->dim() == 1 ? *A_log : A_log->reshape({H});
        if (dt_bias) b = dt_bias->dim() == 1 ? *dt_bias : dt_bias->reshape({H * K});
    }
    sp.scale = scale.value_or(1.0 / std::sqrt((double)K));
    sp.flags = (int)flags;
    sp.output_final_state = output_final_state;
    const Tensor &h = val(h0), &wq = val(cq), &wk = val(ck), &wv = val(cv);
    require_device(q, "k", k); require_device(q, "v", v); require_device(q, "g", g); require_device(q, "beta", beta);
    require_device(q, "A_log", a); require_device(q, "dt_bias", b); require_device(q, "initial_state", h);
    require_device(q, "short_conv_weights[0]", wq); require_device(q, "short_conv_weights[1]", wk);
    require_device(q, "short_conv_weights[2]", wv);
    const std::array<const Tensor*, 11> inputs = {&q, &k, &v, &g, &beta, &a, &b, &h, &wq, &wk, &wv};
    refuse_tangents(inputs);
    bool grad = false;
    if (at::GradMode::is_enabled())
        for (const Tensor* t : inputs) grad = grad || (t->defined() && t->requires_grad());
    c10::cuda::CUDAGuard guard(q.device());
    if (!grad) {
        at::NoGradGuard no_grad;
        FwdOut f = run_fwd(gather(q, k, v, g, beta, a, b, h, wq, wk, wv, tables), sp);
        return {f.o, opt(f.ht)};
    }
    sp.keep = disable_recompute;
    variable_list r = ChunkKda::apply(q, k, v, g, beta, opt(a), opt(b), opt(h), opt(wq), opt(wk), opt(wv), tables, sp);
    return {r[0], r.size() > 1 ? OptTensor(r[1]) : OptTensor()};
}

// ---- the whole sublayer ----------------------------------------------------------------------------------------
// KimiDeltaAttention (k3mini/model.py:132-227) with BF16 activations, d = 128 and the fused short convolution, as one
// autograd node.  The arithmetic is that of the module's parts; what the node saves is around them:
//   * all weights become one BF16 buffer in one launch (autocast would convert them one by one);
//   * q, k, v come from one batched GEMM, and so do the decay and the output gate; the gradients of those weights and
//     the gradient of the two ranks likewise (written where the next GEMM reads them, no concatenation);
//   * weight gradients leave the GEMMs in FP32, the parameters' type, instead of BF16 plus a conversion;
//   * no Python between the launches.
struct LayerSpec {
    Spec op;
    int64_t H = 0;
    double eps = 1e-6;
};
enum { P_WQ, P_WK, P_WV, P_CQ, P_CK, P_CV, P_ALOG, P_FA, P_FB, P_DTB, P_BETA, P_GA, P_GB, P_NORM, P_WO, P_COUNT };
constexpr int64_t HD = 128;

struct Weights { Tensor qkv, narrow, ab, out; };  // views of one BF16 buffer

struct LayerState {
    Inputs in;  // q, k, v, decay, beta and the parameters of the op
    Tensor x2, narrow, gates, o, y, ws, borders, norm_w;
    Weights w;
};

Weights pack_weights(const variable_list& prm, int64_t width, int64_t proj, int64_t H, int64_t wide) {
    const int64_t n_qkv = 3 * proj * width, n_nar = wide * width, n_ab = 2 * proj * HD, n_out = width * proj;
    Tensor buf = at::empty({n_qkv + n_nar + n_ab + n_out}, prm[P_WQ].options().dtype(at::kBFloat16).requires_grad(false));
    char* base = static_cast<char*>(buf.data_ptr());
    KdaPackSegment seg[KDA_PACK_MAX];
    int n = 0;
    int64_t off = 0;
    std::vector<Tensor> hold;  // copies of what is not contiguous FP32 / BF16, until the launch
    auto add = [&](int which, int64_t pad) {
        Tensor t = prm[which];
        if (t.scalar_type() != at::kFloat && t.scalar_type() != at::kBFloat16) t = t.to(at::kFloat);
        if (!t.is_contiguous()) t = t.contiguous();
        hold.push_back(t);
        seg[n++] = {t.data_ptr(), base + 2 * off, t.numel(), pad, t.scalar_type() == at::kFloat ? KDA_DTYPE_F32 : KDA_DTYPE_BF16};
        off += t.numel() + pad;
    };
    for (int i : {P_WQ, P_WK, P_WV, P_FA, P_GA}) add(i, 0);
    add(P_BETA, (wide - 2 * HD - H) * width);
    for (int i : {P_FB, P_GB, P_WO}) add(i, 0);
    check_rc(kda_pack_bf16(seg, n, stream_of(buf)), "kda_pack_bf16");
    Weights w;
    w.qkv = buf.narrow(0, 0, n_qkv).view({3, proj, width});
    w.narrow = buf.narrow(0, n_qkv, n_nar).view({wide, width});
    w.ab = buf.narrow(0, n_qkv + n_nar, n_ab).view({2, proj, HD});
    w.out = buf.narrow(0, n_qkv + n_nar + n_ab, n_out).view({width, proj});
    return w;
}

// the two 128-wide ranks inside the narrow activations as a batch of matrices [2, tokens, 128]
Tensor rank_pair(const Tensor& narrow) {
    return narrow.as_strided({2, narrow.size(0), HD}, {HD, narrow.size(1), 1}, narrow.storage_offset());
}

// The gradients of the two weights behind the ranks, [proj x 128] each, sum over all tokens.  cuBLAS does not split the
// inner dimension of a batch of two, so one CTA per 128 x 128 tile walks every token: 1.2 ns each however many tiles there are
// (up to sixteen heads on 148 SMs).  Cut into pieces the products are bound by their operands, 4 (proj + 128) bytes per token
// at 6.2 TB/s, and cost more launches, partial results and, where the tokens leave a remainder, one more product: some 14 us
// for two to six heads, 20 with a remainder.  The line leaves a margin to that.  Batch against pieces of an eighth (us):
//   tokens            24576        32768        49152        49149        65536       131072
//   1 head          36 : 26      46 : 29      65 : 38      65 : 47      84 : 42     161 : 67
//   6 heads         42 : 40      52 : 46      73 : 58      73 : 63      92 : 71     169 : 108
//   12 heads        51 : 54      63 : 65      84 : 85      84 : 89     103 : 101    184 : 165
//   16 heads        56 : 65      69 : 77      91 : 99      91 : 107    112 : 122    201 : 206
bool rank_cut(int64_t n, int64_t proj) { return n * (1.2 - 4.0 * (proj + HD) / 6200.0) > 26000.0; }

Tensor rank_gradients_cut(const Tensor& dab, const Tensor& narrow) {
    constexpr int64_t CUT = 8;
    const int64_t n = dab.size(1), proj = dab.size(2), wide = narrow.size(1), len = n / CUT, rest = n % CUT;
    const Tensor parts = at::empty({2, CUT + (rest > 0), proj, HD}, dab.options().dtype(at::kFloat));
    for (int i : {0, 1}) {
        Tensor out = parts[i].narrow(0, 0, CUT);
        const Tensor rows = narrow.as_strided({CUT, len, HD}, {len * wide, wide, 1}, narrow.storage_offset() + i * HD);
        at::bmm_out(out, dab[i].narrow(0, 0, CUT * len).view({CUT, len, proj}).transpose(1, 2), rows, at::kFloat);
    }
    if (rest) {
        Tensor out = parts.select(1, CUT);
        at::bmm_out(out, dab.narrow(1, CUT * len, rest).transpose(1, 2), rank_pair(narrow.narrow(0, CUT * len, rest)), at::kFloat);
    }
    return parts.sum(1);
}

Tensor layer_fwd(const Tensor& x, const variable_list& prm, const LayerSpec& ls, const Inputs& tables, LayerState& st, bool recompute = false) {
    const int64_t H = ls.H, proj = H * HD, width = x.size(-1), wide = (2 * HD + H + 7) / 8 * 8;
    const int64_t B = x.size(0), T = x.size(1), n = B * T;
    st.x2 = ready(x, at::kBFloat16).view({n, width});
    st.w = pack_weights(prm, width, proj, H, wide);
    const Tensor qkv = at::bmm(st.x2.unsqueeze(0).expand({3, n, width}), st.w.qkv.transpose(1, 2));
    st.narrow = at::mm(st.x2, st.w.narrow.t());
    const Tensor ab = at::bmm(rank_pair(st.narrow), st.w.ab.transpose(1, 2));
    auto heads = [&](const Tensor& t) { return t.view({B, T, H, HD}); };
    st.gates = ab[1];
    const Tensor beta = st.narrow.narrow(1, 2 * HD, H).contiguous().view({B, T, H});
    st.in = gather(heads(qkv[0]), heads(qkv[1]), heads(qkv[2]), heads(ab[0]), beta, prm[P_ALOG], prm[P_DTB].reshape({proj}), Tensor(),
                   prm[P_CQ], prm[P_CK], prm[P_CV], tables);
    FwdOut f = run_fwd(st.in, ls.op, recompute);
    st.o = f.o;
    st.ws = f.ws;
    st.borders = f.borders;
    st.norm_w = ready(prm[P_NORM], at::kFloat);
    st.y = at::empty({n, proj}, st.x2.options());
    check_rc(kda_norm_gate_fwd(st.o.data_ptr(), st.gates.data_ptr(), ptr<float>(st.norm_w), st.y.data_ptr(), nullptr, n * H, (int)HD,
                               (float)ls.eps, KDA_DTYPE_BF16, stream_of(x)),
             "kda_norm_gate_fwd");
    return at::mm(st.y, st.w.out.t()).view({B, T, width});
}

struct Layer : torch::autograd::Function<Layer> {
    static variable_list forward(AutogradContext* ctx, Tensor x, Tensor p0, Tensor p1, Tensor p2, Tensor p3, Tensor p4, Tensor p5,
                                 Tensor p6, Tensor p7, Tensor p8, Tensor p9, Tensor p10, Tensor p11, Tensor p12, Tensor p13, Tensor p14,
                                 const Inputs& tables, const LayerSpec& ls) {
        const variable_list prm = {p0, p1, p2, p3, p4, p5, p6, p7, p8, p9, p10, p11, p12, p13, p14};
        LayerState st;
        const Tensor out = layer_fwd(x, prm, ls, tables, st, !ls.op.keep);
        variable_list keep = to_list(st.in, ls.op.keep ? st.ws : Tensor(), st.borders);
        for (const Tensor& t : {st.x2, st.narrow, st.gates, st.o, st.y, st.w.qkv, st.w.narrow, st.w.ab, st.w.out, st.norm_w})
            keep.push_back(t);
        ctx->save_for_backward(std::move(keep));
        save_spec(ctx, ls.op);
        ctx->saved_data["eps"] = ls.eps;
        std::vector<int64_t> f32;  // which parameters want a gradient of more than 16 bits
        for (const Tensor& t : prm) f32.push_back(t.element_size() > 2);
        ctx->saved_data["f32"] = f32;
        return {out};
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const variable_list s = ctx->get_saved_variables();
        const Inputs in = from_list(s);
        const Tensor &x2 = s[17], &narrow = s[18], &gates = s[19], &o = s[20], &y = s[21], &norm_w = s[26];
        const Weights w = {s[22], s[23], s[24], s[25]};
        const std::vector<int64_t> f32 = ctx->saved_data["f32"].toIntVector();
        variable_list r(1 + P_COUNT + 2);
        if (!grads[0].defined()) return r;
        c10::cuda::CUDAGuard guard(x2.device());
        const int64_t n = x2.size(0), width = x2.size(1), H = in.q.size(2), proj = H * HD, wide = narrow.size(1);
        const auto bf = x2.options();
        const Tensor dout = ready(grads[0], at::kBFloat16).view({n, width});
        auto need = [&](int which) { return ctx->needs_input_grad(1 + which); };
        // weight gradients straight from the GEMM's FP32 accumulators in FP32 if one of the parameters that share the product
        // has it (the engine rounds the others' shares to their types)
        auto weight_grad = [&](const Tensor& a, const Tensor& b, std::initializer_list<int> which) {
            const bool wide = std::any_of(which.begin(), which.end(), [&](int i) { return f32[i]; });
            if (a.dim() == 3) return wide ? at::bmm(a, b, at::kFloat) : at::bmm(a, b);
            return wide ? at::mm(a, b, at::kFloat) : at::mm(a, b);
        };
        if (need(P_WO)) r[1 + P_WO] = weight_grad(dout.t(), y, {P_WO});
        const Tensor dy = at::mm(dout, w.out);
        // norm and gate
        const Tensor dab = at::empty({2, n, proj}, bf);  // gradients of the decay and of the output gate
        const Tensor d_o = at::empty_like(o);
        constexpr int n_partial = 592;
        const Tensor part = at::empty({n_partial, HD}, bf.dtype(at::kFloat)), dnorm = at::empty({HD}, bf.dtype(at::kFloat));
        check_rc(kda_norm_gate_bwd(o.data_ptr(), gates.data_ptr(), ptr<float>(norm_w), dy.data_ptr(), d_o.data_ptr(), dab[1].data_ptr(),
                                   ptr<float>(dnorm), ptr<float>(part), n_partial, n * H, (int)HD,
                                   (float)ctx->saved_data["eps"].toDouble(), KDA_DTYPE_BF16, stream_of(x2)),
                 "kda_norm_gate_bwd");
        r[1 + P_NORM] = dnorm;
        // the op; its gradients go where the batched GEMMs below read them
        const Tensor dqkv = at::empty({3, n, proj}, bf);
        Grads gr;
        gr.q = dqkv[0]; gr.k = dqkv[1]; gr.v = dqkv[2]; gr.g = dab[0];
        gr = run_bwd(in, load_spec(ctx), s[15], s[16], d_o, Tensor(), gr);
        r[1 + P_CQ] = as_filter(gr.conv_q);
        r[1 + P_CK] = as_filter(gr.conv_k);
        r[1 + P_CV] = as_filter(gr.conv_v);
        r[1 + P_ALOG] = gr.A_log;
        r[1 + P_DTB] = gr.dt_bias.view({H, HD});
        // narrow activations: the two ranks' gradients land in their columns, beta's are copied next to them
        const Tensor dn = at::empty({n, wide}, bf);
        Tensor dn_ranks = rank_pair(dn);
        at::bmm_out(dn_ranks, dab, w.ab);
        dn.narrow(1, 2 * HD, H).copy_(gr.beta.view({n, H}));
        if (wide > 2 * HD + H) dn.narrow(1, 2 * HD + H, wide - 2 * HD - H).zero_();
        if (need(P_FB) || need(P_GB)) {
            const Tensor d = rank_cut(n, proj) ? rank_gradients_cut(dab, narrow)
                                               : weight_grad(dab.transpose(1, 2), rank_pair(narrow), {P_FB, P_GB});
            r[1 + P_FB] = d[0];
            r[1 + P_GB] = d[1];
        }
        if (need(P_FA) || need(P_GA) || need(P_BETA)) {
            const Tensor d = weight_grad(dn.t(), x2, {P_FA, P_GA, P_BETA});
            r[1 + P_FA] = d.narrow(0, 0, HD);
            r[1 + P_GA] = d.narrow(0, HD, HD);
            r[1 + P_BETA] = d.narrow(0, 2 * HD, H);
        }
        if (need(P_WQ) || need(P_WK) || need(P_WV)) {
            const Tensor d = weight_grad(dqkv.transpose(1, 2), x2.unsqueeze(0).expand({3, n, width}), {P_WQ, P_WK, P_WV});
            r[1 + P_WQ] = d[0];
            r[1 + P_WK] = d[1];
            r[1 + P_WV] = d[2];
        }
        if (ctx->needs_input_grad(0)) {  // accumulated inside the GEMMs
            Tensor dx = at::mm(dqkv[0], w.qkv[0]);
            dx.addmm_(dqkv[1], w.qkv[1]);
            dx.addmm_(dqkv[2], w.qkv[2]);
            dx.addmm_(dn, w.narrow);
            r[0] = dx.view({in.q.size(0), in.q.size(1), width});
        }
        return r;
    }
};

// The node derives every size from x and H and hands raw pointers on, so it takes only plain tensors of exactly those sizes
// on x's device.
bool layer_takes(const Tensor& x, const std::vector<Tensor>& prm, int64_t H) {
    if (x.dim() != 3 || prm.size() != P_COUNT || H < 1) return false;
    for (const Tensor& t : prm)
        if (t.device() != x.device() || t.layout() != at::kStrided || t.unsafeGetTensorImpl()->is_python_dispatch()) return false;
    const int64_t width = x.size(2), proj = H * HD, ksize = prm[P_CQ].dim() == 3 ? prm[P_CQ].size(2) : 0;
    if (ksize < 1 || ksize > 4) return false;
    auto is = [&](int which, at::IntArrayRef sizes) { return prm[which].sizes() == sizes; };
    for (int i : {P_WQ, P_WK, P_WV})
        if (!is(i, {proj, width})) return false;
    for (int i : {P_CQ, P_CK, P_CV})
        if (!is(i, {proj, 1, ksize})) return false;
    for (int i : {P_FA, P_GA})
        if (!is(i, {HD, width})) return false;
    for (int i : {P_FB, P_GB})
        if (!is(i, {proj, HD})) return false;
    return is(P_ALOG, {H}) && is(P_DTB, {H, HD}) && is(P_BETA, {H, width}) && is(P_NORM, {HD}) && is(P_WO, {width, proj});
}

// nothing where the node does not take these tensors: the module's parts then compute what they can, or say what is wrong
OptTensor layer(const Tensor& x, const std::vector<Tensor>& prm, int64_t H, double scale, double eps, bool disable_recompute,
                OptTensor cu, OptTensor chunk_seq, OptTensor seq_off, OptTensor chunk_tab, int64_t NT, int64_t longest) {
    require_cuda(x);
    if (!layer_takes(x, prm, H)) return std::nullopt;
    LayerSpec ls;
    ls.H = H;
    ls.eps = eps;
    ls.op.scale = scale;
    ls.op.flags = KDA_FLAG_QK_L2NORM | KDA_FLAG_GATE | KDA_FLAG_BETA_SIGMOID | KDA_FLAG_STATE_V_FIRST;
    ls.op.longest = longest;
    ls.op.NT = cu ? NT : x.size(0) * ((x.size(1) + CHUNK - 1) / CHUNK);
    Inputs tables;
    if (cu) take_tables(tables, cu, chunk_seq, seq_off, chunk_tab, x.size(0));
    std::array<const Tensor*, 1 + P_COUNT> inputs = {&x};
    for (int i = 0; i < P_COUNT; ++i) inputs[1 + i] = &prm[i];
    refuse_tangents(inputs);
    bool grad = false;
    if (at::GradMode::is_enabled())
        for (const Tensor* t : inputs) grad = grad || t->requires_grad();
    c10::cuda::CUDAGuard guard(x.device());
    // the node does its own conversions; autocast must not see its matrix products
    c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::autocast_dispatch_keyset);
    if (!grad) {
        at::NoGradGuard no_grad;
        LayerState st;
        return layer_fwd(x, prm, ls, tables, st);
    }
    ls.op.keep = disable_recompute;
    return Layer::apply(x, prm[0], prm[1], prm[2], prm[3], prm[4], prm[5], prm[6], prm[7], prm[8], prm[9], prm[10], prm[11], prm[12],
                        prm[13], prm[14], tables, ls)[0];
}

}  // namespace

PYBIND11_MODULE(_host, m) {
    m.def("set_status", &set_status);
    m.def("set_callbacks", &set_callbacks);
    m.def("env_flags", &env_flags);
    // allocations and launches may wait for the device, so other Python threads run meanwhile
    const py::call_guard<py::gil_scoped_release> unlocked;
    m.def("recurrent", &recurrent, unlocked);
    m.def("chunk_kda", &chunk_kda, unlocked);
    m.def("layer", &layer, unlocked);
    m.def("layer_takes", &layer_takes);
}
