// Host path of the torch front end: argument checks, dtype policy, output allocation, autograd wiring and the calls
// into the C ABI, in native code.
//
// A single-token step or a short prompt keeps the GPU busy for a few microseconds, so what such a call costs is the
// host work in front of the launch.  With the checks, ctypes structs and Python-registered operators that work took
// 50 us for one decode step; here it is a few microseconds plus the launches.
//
// Two ways in:
//   * run(), decode_step(), layer_*(): what the Python functions call.  Plain CUDA tensors with nothing in between go
//     straight to the implementation (with one autograd node where gradients are wanted); for anything else run() and
//     decode_step() hand NotImplemented back, and the Python functions go through the operators.
//   * torch.ops.palimpsa_b200.{fwd, bwd, decode_step}: the registered operators, which tracing, functorch and
//     fake-tensor modes see.  Same implementation underneath; their fake kernels are registered from Python.
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/record_function.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/autograd_not_implemented_fallback.h>
#include <torch/extension.h>
#include <torch/library.h>

#include <array>
#include <optional>
#include <tuple>

#include "../../include/palimpsa_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

// ---- small helpers ------------------------------------------------------------------------------------
void check_rc(int rc, const char* what) {
    TORCH_CHECK(rc == PALIMPSA_OK, what, " failed with code ", rc, ": ", palimpsa_last_error_string(rc));
}
bool supported_dtype(at::ScalarType t) { return t == at::kFloat || t == at::kBFloat16 || t == at::kHalf; }
int io_code(at::ScalarType t) {
    TORCH_CHECK_TYPE(supported_dtype(t), "unsupported dtype ", t, "; use float32, bfloat16 or float16");
    return t == at::kFloat ? PALIMPSA_F32 : (t == at::kBFloat16 ? PALIMPSA_BF16 : PALIMPSA_F16);
}
Tensor empty(at::IntArrayRef sizes, at::ScalarType dt, const at::Device& dev) {
    return at::detail::empty_cuda(sizes, dt, dev, std::nullopt);
}
Tensor none_like(const Tensor& t, at::ScalarType dt) { return at::empty({0}, t.options().dtype(dt)); }
template <class T = void>
T* ptr(const Tensor& t) {
    return t.defined() && t.numel() ? static_cast<T*>(const_cast<void*>(t.const_data_ptr())) : nullptr;
}
template <class T = void>
T* ptr(const OptTensor& t) {
    return t ? ptr<T>(*t) : nullptr;
}
bool given(const OptTensor& t) { return t.has_value() && t->defined(); }
void require_cuda(std::initializer_list<const Tensor*> ts) {
    for (const Tensor* t : ts)
        TORCH_CHECK(!t->defined() || t->is_cuda(),
                    "palimpsa_b200 runs on CUDA (sm_100a) only and has no CPU path; for CPU tensors use "
                    "palimpsa_b200.ops.palimpsa_ref (naive recurrence).");
}
// The last check before pointers are taken, whichever way a call came in: the kernels read each argument through a raw
// pointer, so a host tensor, one of another GPU, another dtype, length or stride would be a fault or garbage there.
void check_arg(const char* name, const Tensor& t, at::ScalarType dt, at::IntArrayRef sizes, const at::Device& dev) {
    if (!t.defined()) return;
    require_cuda({&t});
    TORCH_CHECK_VALUE(t.device() == dev, name, " is on ", t.device(), ", q on ", dev);
    TORCH_CHECK_TYPE(t.scalar_type() == dt, name, " has dtype ", t.scalar_type(), ", expected ", dt);
    TORCH_CHECK_VALUE(t.numel() == c10::multiply_integers(sizes), name, " has shape ", t.sizes(), ", expected ", sizes);
    TORCH_CHECK_VALUE(t.is_contiguous(), name, " is not contiguous");
}
// Nothing between the caller and the kernels: dense CUDA tensors and the thread's usual dispatch state.  Everything else
// (a mode, a transform, a tracer, a fake, negated, batched or wrapped tensor, a kernel that runs below autograd) has a
// dispatch key of its own, on the thread or on the tensor, and goes through the registered operators, which is where those
// hook in.  Named by what is allowed, so that a key nobody thought of takes the general route.
bool plain(std::initializer_list<const Tensor*> ts) {
    using c10::DispatchKey;
    using c10::DispatchKeySet;
    // bits, not key-set differences: those leave a set's backends standing
    static const uint64_t usual_state = (c10::default_included_set | c10::autocast_dispatch_keyset).raw_repr();
    static const uint64_t usual_tensor = (DispatchKeySet(DispatchKey::CUDA) | DispatchKeySet(DispatchKey::AutogradCUDA) |
                                          DispatchKeySet(DispatchKey::ADInplaceOrView) | DispatchKeySet(DispatchKey::AutocastCUDA))
                                             .raw_repr();
    if (c10::impl::dispatch_mode_enabled()) return false;
    const c10::impl::LocalDispatchKeySet tls = c10::impl::tls_local_dispatch_key_set();
    if (tls.included_.raw_repr() & ~usual_state) return false;
    // below autograd no node may be made (inference mode is there too, with gradients off: nothing to make)
    if (at::GradMode::is_enabled() && (tls.excluded_.raw_repr() & c10::autograd_dispatch_keyset.raw_repr())) return false;
    for (const Tensor* t : ts)
        if (t->defined() && (t->key_set().raw_repr() & ~usual_tensor)) return false;
    return true;
}
py::object not_plain() { return py::reinterpret_borrow<py::object>(Py_NotImplemented); }  // the caller takes the general route
Tensor as(const Tensor& t, at::ScalarType dt) {
    Tensor r = t.scalar_type() == dt ? t : t.to(dt);
    return r.is_contiguous() ? r : r.contiguous();
}
Tensor as_opt(const OptTensor& t, at::ScalarType dt) { return given(t) ? as(*t, dt) : Tensor(); }
Tensor dense(const Tensor& t) { return t.is_contiguous() ? t : t.contiguous(); }
Tensor dense(const OptTensor& t) { return given(t) ? dense(*t) : Tensor(); }
void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

int sm_count(const OptTensor& t) {
    if (!given(t) || !t->is_cuda()) return at::cuda::is_available() ? at::cuda::getCurrentDeviceProperties()->multiProcessorCount : 148;
    return at::cuda::getDeviceProperties(t->get_device())->multiProcessorCount;
}

// ---- segments ---------------------------------------------------------------------------------------------
int64_t segment_len(int64_t T, int64_t G) {
    const int64_t per = (T + G - 1) / G, CI = PALIMPSA_CKPT_INTERVAL;
    return std::max<int64_t>(CI, (per + CI - 1) / CI * CI);
}

// Does cutting this problem round what crosses a boundary to bfloat16?  The summary and the carried-gradient kernels on the
// tensor cores do (their shapes: bf16, d_v <= 128, d_k and d_v multiples of 8, padded d_k 32 to 128; the summary from 8192
// state elements per head, the carried terms without the uncertainty output); all other passes are exact float32.
bool boundaries_rounded(int64_t K, int64_t V, int io, bool unc) {
    const int64_t KP = palimpsa_padded_k((int)K);
    return io == PALIMPSA_BF16 && V <= 128 && V % 8 == 0 && K % 8 == 0 && KP >= 32 && KP <= 128 && (!unc || KP * V >= 8192);
}
// CTAs per sequence-head at fixed tile heights: 8 warps (4 where d_v is short), 6 at d_k = 48 and 11 or 12 at d_k = 128 by
// which pads d_v less.  Only what is starved of CTAs at these is ever rounded: which calls keep float32 boundaries must not
// change whenever the tile heights are tuned.
int64_t nominal_tiles(int64_t K, int64_t V) {
    const int64_t KP = palimpsa_padded_k((int)K), per_warp = KP <= 48 ? 8 : KP <= 96 ? 4 : 2;
    const auto up = [V](int64_t rows) { return (V + rows - 1) / rows * rows; };
    int64_t warps = V > 4 * per_warp ? 8 : 4;
    if (KP == 128 && V >= 48) warps = up(22) < up(24) ? 11 : 12;
    if (KP == 48 && warps == 8 && up(48) < up(64)) warps = 6;
    return up(warps * per_warp) / (warps * per_warp);
}

// How many segments to cut every sequence into on one GPU (plan_segments in _core.py documents the rule).
int64_t plan_segments(int64_t N, int64_t T, int64_t H, int64_t K, int64_t V, int64_t sms, bool backward, int io, bool unc,
                      bool packed) {
    const bool shorter = T < 2048;
    if (shorter && (T < 256 || packed || io == PALIMPSA_BF16)) return 1;
    const int64_t rows = palimpsa_fwd_tile_rows((int)K, (int)V);
    TORCH_CHECK_VALUE(rows > 0, "d_k = ", K, " is above the supported maximum of 256");
    const int64_t pieces = std::max<int64_t>(1, std::min<int64_t>(32, T / 256));
    if (!backward) {
        const int64_t ctas = N * H * ((V + rows - 1) / rows);
        if (shorter) {
            const int64_t G = std::min<int64_t>(T / 64, sms / std::max<int64_t>(ctas, 1));
            return G >= 3 ? G : 1;
        }
        return ctas >= sms ? 1 : pieces;
    }
    const int64_t brow = palimpsa_bwd_tile_rows((int)K, (int)V, io, unc ? 1 : 0);
    TORCH_CHECK_VALUE(brow > 0, "no backward tiling for d_k = ", K, ", d_v = ", V);
    const int64_t ctas = N * H * ((V + brow - 1) / brow);
    const bool rounded = boundaries_rounded(K, V, io, unc);
    const int64_t nominal = N * H * nominal_tiles(K, V);
    if (packed) return ctas >= sms || (rounded && nominal >= sms) ? 1 : pieces;
    palimpsa_problem p{};
    p.num_seqs = (int)N, p.seq_len = (int)T, p.H = (int)H, p.K = (int)K, p.V = (int)V, p.io_dtype = io;
    p.flags = unc ? PALIMPSA_FLAG_UNCERTAINTY : 0;
    const double uncut = palimpsa_bwd_token_cost(&p);
    if (shorter) {  // one wave of segments; a segment's backward takes its state-gradient pass first
        const int64_t G = std::min<int64_t>(T / 64, sms / std::max<int64_t>(ctas, 1));
        p.num_seqs = 0;  // per CTA of a full grid
        const double one_wave = palimpsa_bwd_token_cost(&p) * (double)sms / (double)((V + brow - 1) / brow);
        return G >= 2 && (double)T * uncut > 1.6 * one_wave * (double)T / (double)G + 400 ? G : 1;
    }
    if (rounded && 10 * nominal >= 8 * ((nominal + sms - 1) / sms) * sms) return 1;
    if (pieces < 2) return 1;
    p.segments = (int)pieces;
    // How much cheaper the cut backward has to be: less where its uncut grid is one wave (that of 4 warps below 9 units, any
    // below 15) and the forward's leaves SMs idle too, so that the summaries and the scan are paid for there.
    const bool one = uncut < 15;
    const double worth = rounded ? (one ? 1.05 : 1.15) : K <= 16 || uncut < 9 ? 1.2 : one ? 1.25 : 1.55;
    return uncut > worth * palimpsa_bwd_token_cost(&p) ? pieces : 1;
}

// The [N,G,H,V,KP] boundary buffers of a segmented pass, in one allocation (returned as its owner).
Tensor segment_buffers(palimpsa_segments& sg, int64_t N, int64_t G, int64_t T, int64_t H, int64_t V, int64_t K, bool fwd,
                       const at::Device& dev) {
    const int64_t n = N * G * H * V * palimpsa_padded_k((int)K);  // a multiple of 16 floats
    sg = palimpsa_segments{};
    sg.num_segments = (int)G;
    sg.seg_len = (int)segment_len(T, G);
    Tensor buf = empty({4 * n}, at::kFloat, dev);
    float* p = ptr<float>(buf);
    if (fwd) {
        sg.sum_M = p, sg.sum_J = p + n, sg.start_M = p + 2 * n, sg.start_I = p + 3 * n;
    } else {
        sg.carry_M = p, sg.carry_I = p + n, sg.rloc_M = p + 2 * n, sg.rloc_I = p + 3 * n;
    }
    return buf;
}

// ---- the operator, forward and backward -------------------------------------------------------------------
palimpsa_problem make_problem(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b, const Tensor& gt,
                              const Tensor& g, const Tensor& Ip, const Tensor& cu, const Tensor& coff, const Tensor& order,
                              const Tensor& mu0, const Tensor& I0, double scale, int flags) {
    palimpsa_problem p{};
    const int64_t B = q.size(0), T = q.size(1);
    const bool packed = cu.defined();
    p.num_seqs = (int)(packed ? cu.numel() - 1 : B);
    p.seq_len = (int)(packed ? 0 : T);
    p.total_tokens = (int)(B * T);
    p.H = (int)q.size(2), p.K = (int)q.size(3), p.V = (int)v.size(3);
    p.io_dtype = io_code(q.scalar_type());
    p.flags = flags;
    p.scale = (float)scale;
    p.q = ptr(q), p.k = ptr(k), p.v = ptr(v), p.b = ptr(b);
    p.gt = ptr<float>(gt), p.g = ptr<float>(g), p.Ip = ptr<float>(Ip);
    p.cu_seqlens = ptr<int32_t>(cu), p.chunk_offsets = ptr<int32_t>(coff), p.seq_order = ptr<int32_t>(order);
    p.init_mu = ptr<float>(mu0), p.init_I = ptr<float>(I0);
    return p;
}

struct Inputs {
    Tensor q, k, v, b, gt, g, Ip;
    Tensor mu0, I0, cu;  // undefined where absent
};
struct Options {
    double scale = 1.0;
    bool unc = false, save_ckpt = false, want_final = false, recurrent = false, carry_tc = true;
    int64_t segments = 1;
};
struct FwdOut {
    Tensor o, o_var, fmu, fI, ckM, ckI, coff, order, decay;  // undefined where not asked for
};

void check_inputs(const Inputs& x) {
    TORCH_CHECK_VALUE(x.q.dim() == 4 && x.k.sizes() == x.q.sizes() && x.v.dim() == 4 && x.b.sizes() == x.v.sizes() &&
                          x.v.sizes().slice(0, 3) == x.q.sizes().slice(0, 3),
                      "expected q,k [B,T,H,K] and v,b [B,T,H,V]");
    const int64_t B = x.q.size(0), T = x.q.size(1), H = x.q.size(2), K = x.q.size(3), V = x.v.size(3);
    const at::Device dev = x.q.device();
    const at::ScalarType io = x.q.scalar_type();
    io_code(io);
    check_arg("q", x.q, io, {B, T, H, K}, dev);
    check_arg("k", x.k, io, {B, T, H, K}, dev);
    check_arg("v", x.v, io, {B, T, H, V}, dev);
    check_arg("b", x.b, io, {B, T, H, V}, dev);
    check_arg("gt", x.gt, at::kFloat, {B, T, H}, dev);
    check_arg("g", x.g, at::kFloat, {H}, dev);
    check_arg("Ip", x.Ip, at::kFloat, {H}, dev);
    if (x.cu.defined()) {
        TORCH_CHECK_VALUE(B == 1 && x.cu.numel() >= 1, "cu_seqlens [N+1] goes with one packed row");
        check_arg("cu_seqlens", x.cu, at::kInt, {x.cu.numel()}, dev);
    }
    const int64_t N = x.cu.defined() ? x.cu.numel() - 1 : B;
    TORCH_CHECK_VALUE(x.mu0.defined() == x.I0.defined(), "initial_mu_state and initial_I_state must be given together");
    check_arg("initial_mu_state", x.mu0, at::kFloat, {N, H, V, K}, dev);
    check_arg("initial_I_state", x.I0, at::kFloat, {N, H, V, K}, dev);
}

FwdOut fwd_impl(const Inputs& x, const Options& opt) {
    check_inputs(x);
    const int64_t B = x.q.size(0), T = x.q.size(1), H = x.q.size(2), K = x.q.size(3), V = x.v.size(3);
    const int64_t N = x.cu.defined() ? x.cu.numel() - 1 : B;
    const at::Device dev = x.q.device();
    c10::cuda::CUDAGuard guard(dev);
    void* st = stream_of(x.q);
    FwdOut r;
    r.o = empty({B, T, H, V}, x.q.scalar_type(), dev);
    if (opt.unc) r.o_var = empty({B, T, H, V}, x.q.scalar_type(), dev);
    if (opt.want_final) {
        r.fmu = empty({N, H, V, K}, at::kFloat, dev);
        r.fI = empty({N, H, V, K}, at::kFloat, dev);
    }
    if (x.cu.defined()) {  // checkpoint slots of the documents, and the order to start them in (longest first)
        Tensor plan = empty({2 * N}, at::kInt, dev);
        r.coff = plan.narrow(0, 0, N);
        r.order = plan.narrow(0, N, N);
        check_rc(palimpsa_varlen_plan(ptr<int32_t>(x.cu), (int)N, ptr<int32_t>(r.coff), ptr<int32_t>(r.order), st),
                 "palimpsa packed-batch plan");
    }
    if (opt.save_ckpt) {
        const int64_t slots = (B * T + PALIMPSA_CKPT_INTERVAL - 1) / PALIMPSA_CKPT_INTERVAL + N, KP = palimpsa_padded_k((int)K);
        r.ckM = empty({slots, H, V, KP}, at::kFloat, dev);
        r.ckI = empty({slots, H, V, KP}, at::kFloat, dev);
    }
    palimpsa_fwd_params prm{};
    prm.struct_size = sizeof(prm);
    prm.p = make_problem(x.q, x.k, x.v, x.b, x.gt, x.g, x.Ip, x.cu, r.coff, r.order, x.mu0, x.I0, opt.scale,
                         opt.unc ? PALIMPSA_FLAG_UNCERTAINTY : 0);
    prm.o = ptr(r.o), prm.o_var = ptr(r.o_var);
    prm.final_mu = ptr<float>(r.fmu), prm.final_I = ptr<float>(r.fI);
    prm.ckpt_M = ptr<float>(r.ckM), prm.ckpt_I = ptr<float>(r.ckI);
    if (opt.segments > 1 && T > 0) {
        // summaries of every segment -> boundary scan -> all segments run side by side; in a packed batch (T = all
        // tokens) a segment index beyond a sequence's end is an empty segment
        palimpsa_segments sg;
        Tensor bufs = segment_buffers(sg, N, opt.segments, T, H, V, K, true, dev);
        r.decay = empty({N, opt.segments, H}, at::kFloat, dev);
        sg.decay = ptr<float>(r.decay);
        check_rc(palimpsa_segment_summary(&prm.p, &sg, st), "palimpsa segment summary");
        check_rc(palimpsa_cp_combine(&prm.p, &sg, nullptr, nullptr, nullptr, nullptr, st), "palimpsa boundary scan");
        check_rc(palimpsa_chunk_fwd_segments(&prm, &sg, st), "palimpsa forward (segments)");
    } else {
        check_rc(opt.recurrent ? palimpsa_recurrent_fwd(&prm, st) : palimpsa_chunk_fwd(&prm, st), "palimpsa forward");
    }
    return r;
}

struct BwdIn {
    Tensor d_o, d_o_var;  // d_o_var undefined without the uncertainty output
    Tensor coff, order, ckM, ckI, decay;
    bool explicit_init = false, recurrent = false, carry_tc = true;
    double scale = 1.0;
};
struct BwdOut {
    Tensor dq, dk, dv, db, dgt, dg, dIp;
};

BwdOut bwd_impl(const Inputs& x, const BwdIn& in) {
    check_inputs(x);
    const int64_t B = x.q.size(0), T = x.q.size(1), H = x.q.size(2), K = x.q.size(3), V = x.v.size(3);
    const at::Device dev = x.q.device();
    const at::ScalarType io = x.q.scalar_type();
    const int64_t seqs = x.cu.defined() ? x.cu.numel() - 1 : B;
    check_arg("the gradient of o", in.d_o, io, {B, T, H, V}, dev);
    check_arg("the gradient of o_var", in.d_o_var, io, {B, T, H, V}, dev);
    TORCH_CHECK_VALUE(in.ckM.dim() == 4, "ckpt_M, ckpt_I [slots,H,V,KP]");
    const int64_t slots = in.ckM.size(0), need_slots = (B * T + PALIMPSA_CKPT_INTERVAL - 1) / PALIMPSA_CKPT_INTERVAL + seqs;
    TORCH_CHECK_VALUE(slots >= need_slots, "ckpt_M has ", slots, " slots, expected ", need_slots);
    check_arg("ckpt_M", in.ckM, at::kFloat, {slots, H, V, palimpsa_padded_k((int)K)}, dev);
    check_arg("ckpt_I", in.ckI, at::kFloat, {slots, H, V, palimpsa_padded_k((int)K)}, dev);
    if (x.cu.defined()) {
        TORCH_CHECK_VALUE(in.coff.defined(), "a packed backward needs the forward's chunk_offsets");
        check_arg("chunk_offsets", in.coff, at::kInt, {seqs}, dev);
        check_arg("seq_order", in.order, at::kInt, {seqs}, dev);
    }
    if (in.decay.defined() && in.decay.numel() > 0) {
        TORCH_CHECK_VALUE(in.decay.dim() == 3, "seg_decay [N,G,H]");
        check_arg("seg_decay", in.decay, at::kFloat, {seqs, in.decay.size(1), H}, dev);
    }
    c10::cuda::CUDAGuard guard(dev);
    void* st = stream_of(x.q);
    BwdOut r;
    r.dq = empty({B, T, H, K}, io, dev);
    r.dk = empty({B, T, H, K}, io, dev);
    r.dv = empty({B, T, H, V}, io, dev);
    r.db = empty({B, T, H, V}, io, dev);
    r.dgt = empty({B, T, H}, at::kFloat, dev);
    r.dg = empty({H}, at::kFloat, dev);
    r.dIp = empty({H}, at::kFloat, dev);
    const bool unc = in.d_o_var.defined();
    palimpsa_bwd_params prm{};
    prm.struct_size = sizeof(prm);
    prm.p = make_problem(x.q, x.k, x.v, x.b, x.gt, x.g, x.Ip, x.cu, in.coff, in.order, Tensor(), Tensor(), in.scale,
                         (unc ? PALIMPSA_FLAG_UNCERTAINTY : 0) | (in.explicit_init ? PALIMPSA_FLAG_EXPLICIT_INIT : 0));
    if (in.decay.defined() && in.decay.numel() > 0) prm.p.segments = (int)in.decay.size(1);
    Tensor plan;  // the order to start the documents in, where the forward's was not kept (the operators have no output for it)
    if (x.cu.defined() && !in.order.defined() && seqs > 0) {
        plan = empty({2 * seqs}, at::kInt, dev);
        check_rc(palimpsa_varlen_plan(ptr<int32_t>(x.cu), (int)seqs, ptr<int32_t>(plan), ptr<int32_t>(plan) + seqs, st),
                 "palimpsa packed-batch plan");
        prm.p.seq_order = ptr<int32_t>(plan) + seqs;
    }
    prm.d_o = ptr(in.d_o), prm.d_o_var = ptr(in.d_o_var);
    prm.ckpt_M = ptr<float>(in.ckM), prm.ckpt_I = ptr<float>(in.ckI);
    prm.dq = ptr(r.dq), prm.dk = ptr(r.dk), prm.dv = ptr(r.dv), prm.db = ptr(r.db);
    prm.dgt = ptr<float>(r.dgt), prm.dg = ptr<float>(r.dg), prm.dIp = ptr<float>(r.dIp);
    Tensor ws = empty({std::max<int64_t>((int64_t)palimpsa_bwd_workspace_bytes(&prm.p), 256)}, at::kByte, dev);
    prm.workspace = ptr(ws), prm.workspace_bytes = (size_t)ws.numel();
    if (in.decay.defined() && in.decay.numel() > 0) {
        const int64_t N = x.cu.defined() ? x.cu.numel() - 1 : B, G = in.decay.size(1);
        palimpsa_segments sg;
        Tensor bufs = segment_buffers(sg, N, G, T, H, V, K, false, dev);
        sg.decay = ptr<float>(in.decay);
        if (in.carry_tc && palimpsa_carry_apply_supported(&prm.p)) {
            // zero-carry backward of every segment -> reverse boundary scan -> carried terms on the tensor cores ->
            // finishing kernels
            check_rc(palimpsa_chunk_bwd_segments(&prm, &sg, 2, st), "palimpsa backward (main)");
            check_rc(palimpsa_cp_combine_bwd(&prm.p, &sg, nullptr, nullptr, nullptr, nullptr, st),
                     "palimpsa boundary scan (backward)");
            check_rc(palimpsa_carry_apply(&prm, &sg, st), "palimpsa carried-gradient terms");
            check_rc(palimpsa_chunk_bwd_segments(&prm, &sg, 3, st), "palimpsa backward (finish)");
        } else {
            // state-gradient pass per segment -> reverse boundary scan -> full backward per segment
            check_rc(palimpsa_chunk_bwd_segments(&prm, &sg, 1, st), "palimpsa backward (carry pass)");
            check_rc(palimpsa_cp_combine_bwd(&prm.p, &sg, nullptr, nullptr, nullptr, nullptr, st),
                     "palimpsa boundary scan (backward)");
            sg.rloc_M = sg.rloc_I = nullptr;
            check_rc(palimpsa_chunk_bwd_segments(&prm, &sg, 0, st), "palimpsa backward (segments)");
        }
    } else {
        check_rc(in.recurrent ? palimpsa_recurrent_bwd(&prm, st) : palimpsa_chunk_bwd(&prm, st), "palimpsa backward");
    }
    return r;
}

// ---- registered operators (what tracing and the transforms see) ---------------------------------------------
using FwdTuple = std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor>;
using BwdTuple = std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor>;

FwdTuple fwd_cuda(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b, const Tensor& gt, const Tensor& g,
                  const Tensor& Ip, const OptTensor& init_mu, const OptTensor& init_I, const OptTensor& cu_seqlens,
                  double scale, bool uncertainty, bool save_ckpt, bool want_final, bool recurrent, int64_t num_segments) {
    Options opt;
    opt.scale = scale, opt.unc = uncertainty, opt.save_ckpt = save_ckpt, opt.want_final = want_final;
    opt.recurrent = recurrent, opt.segments = num_segments;
    FwdOut r = fwd_impl({dense(q), dense(k), dense(v), dense(b), dense(gt), dense(g), dense(Ip), as_opt(init_mu, at::kFloat),
                         as_opt(init_I, at::kFloat), as_opt(cu_seqlens, at::kInt)}, opt);
    auto f = [&](Tensor& t, at::ScalarType dt) { return t.defined() ? t : none_like(q, dt); };
    // the slots are handed out as a tensor of their own: an operator's outputs share no storage
    return {r.o, f(r.o_var, q.scalar_type()), f(r.fmu, at::kFloat), f(r.fI, at::kFloat), f(r.ckM, at::kFloat),
            f(r.ckI, at::kFloat), r.coff.defined() ? r.coff.clone() : none_like(q, at::kInt), f(r.decay, at::kFloat)};
}

// palimpsa_b200.ops.palimpsa._core.carry_on_tensor_cores, for calls that come in as a registered operator (the Python
// functions hand it over).  Those come without the interpreter lock.
bool carry_switch() {
    if (!Py_IsInitialized()) return true;
    py::gil_scoped_acquire gil;
    return py::module_::import("palimpsa_b200.ops.palimpsa._core").attr("carry_on_tensor_cores").cast<bool>();
}

BwdTuple bwd_cuda(const Tensor& d_o, const OptTensor& d_o_var, const Tensor& q, const Tensor& k, const Tensor& v,
                  const Tensor& b, const Tensor& gt, const Tensor& g, const Tensor& Ip, const OptTensor& cu_seqlens,
                  const OptTensor& chunk_offsets, const Tensor& ckpt_M, const Tensor& ckpt_I, double scale,
                  bool explicit_init, bool recurrent, const OptTensor& seg_decay) {
    Inputs x{dense(q), dense(k), dense(v), dense(b), dense(gt), dense(g), dense(Ip), Tensor(), Tensor(), as_opt(cu_seqlens, at::kInt)};
    BwdIn in;
    in.d_o = dense(d_o), in.d_o_var = dense(d_o_var);
    in.coff = dense(chunk_offsets);
    in.ckM = dense(ckpt_M), in.ckI = dense(ckpt_I), in.decay = dense(seg_decay);
    in.explicit_init = explicit_init, in.recurrent = recurrent, in.scale = scale;
    if (in.decay.defined() && in.decay.numel() > 0) in.carry_tc = carry_switch();
    BwdOut r = bwd_impl(x, in);
    return {r.dq, r.dk, r.dv, r.db, r.dgt, r.dg, r.dIp};
}

FwdTuple call_fwd_op(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b, const Tensor& gt, const Tensor& g,
                     const Tensor& Ip, const OptTensor& mu0, const OptTensor& I0, const OptTensor& cu, double scale, bool unc,
                     bool save_ckpt, bool want_final, bool recurrent, int64_t segments) {
    static auto op = c10::Dispatcher::singleton().findSchemaOrThrow("palimpsa_b200::fwd", "").typed<decltype(fwd_cuda)>();
    return op.call(q, k, v, b, gt, g, Ip, mu0, I0, cu, scale, unc, save_ckpt, want_final, recurrent, segments);
}
BwdTuple call_bwd_op(const Tensor& d_o, const OptTensor& d_o_var, const Tensor& q, const Tensor& k, const Tensor& v,
                     const Tensor& b, const Tensor& gt, const Tensor& g, const Tensor& Ip, const OptTensor& cu,
                     const OptTensor& coff, const Tensor& ckM, const Tensor& ckI, double scale, bool explicit_init,
                     bool recurrent, const OptTensor& decay) {
    static auto op = c10::Dispatcher::singleton().findSchemaOrThrow("palimpsa_b200::bwd", "").typed<decltype(bwd_cuda)>();
    return op.call(d_o, d_o_var, q, k, v, b, gt, g, Ip, cu, coff, ckM, ckI, scale, explicit_init, recurrent, decay);
}

// What the autograd node keeps besides the saved tensors, as one number and one set of bits: values that hash, which is
// what compiled autograd asks of a node's state.
enum NodeBits : int64_t { NODE_UNC = 1, NODE_RECURRENT = 2, NODE_INIT = 4, NODE_CKPT = 8, NODE_CARRY_TC = 16, NODE_PACKED = 32,
                          NODE_CUT = 64, NODE_IO_SHIFT = 8 };

// Gradients reaching the final states are ignored and initial states get none, as in the reference
// (chunk_palimpsa_forgetting_scalar.py:522, :617-620: truncated BPTT across calls).  Gradients of the other outputs are
// not materialised: autograd would fill a zero tensor for each checkpoint buffer (1.6 GB per step at the benchmark's size).
variable_list node_backward(AutogradContext* ctx, const variable_list& grads, size_t num_inputs) {
    auto saved = ctx->get_saved_variables();
    const int64_t bits = ctx->saved_data["bits"].toInt();
    const auto is = [bits](int64_t bit) { return (bits & bit) != 0; };
    const at::ScalarType io = static_cast<at::ScalarType>(bits >> NODE_IO_SHIFT);
    TORCH_CHECK(is(NODE_CKPT), "palimpsa_b200: backward needs the forward's checkpoints (forward ran with save_ckpt=False)");
    Inputs x{saved[0], saved[1], saved[2], saved[3], saved[4], saved[5], saved[6], Tensor(), Tensor(), is(NODE_PACKED) ? saved[7] : Tensor()};
    BwdIn in;
    in.d_o = grads[0].defined() ? as(grads[0], io) : at::zeros_like(x.v, x.v.options().dtype(io));
    if (is(NODE_UNC)) in.d_o_var = grads[1].defined() ? as(grads[1], io) : at::zeros_like(in.d_o);
    if (is(NODE_PACKED)) in.coff = saved[8], in.order = saved[12];
    in.ckM = saved[9], in.ckI = saved[10];
    if (is(NODE_CUT)) in.decay = saved[11];
    in.explicit_init = is(NODE_INIT), in.recurrent = is(NODE_RECURRENT), in.carry_tc = is(NODE_CARRY_TC);
    in.scale = ctx->saved_data["scale"].toDouble();
    variable_list out(num_inputs);
    // create_graph=True and traced backwards go through the registered operator
    if (at::GradMode::is_enabled() || !plain({&x.q, &x.v, &in.d_o, &in.ckM})) {
        auto opt = [](const Tensor& t) { return t.defined() ? OptTensor(t) : std::nullopt; };
        std::tie(out[0], out[1], out[2], out[3], out[4], out[5], out[6]) =
            call_bwd_op(in.d_o, opt(in.d_o_var), x.q, x.k, x.v, x.b, x.gt, x.g, x.Ip, opt(x.cu), opt(in.coff), in.ckM, in.ckI,
                        in.scale, in.explicit_init, in.recurrent, opt(in.decay));
        return out;
    }
    RECORD_FUNCTION("palimpsa_b200::bwd", c10::ArrayRef<const c10::IValue>{});
    BwdOut r = bwd_impl(x, in);
    out[0] = r.dq, out[1] = r.dk, out[2] = r.dv, out[3] = r.db, out[4] = r.dgt, out[5] = r.dg, out[6] = r.dIp;
    return out;
}
void node_save(AutogradContext* ctx, const Inputs& x, const Tensor& coff, const Tensor& order, const Tensor& ckM,
               const Tensor& ckI, const Tensor& decay, const Options& opt) {
    ctx->save_for_backward({x.q, x.k, x.v, x.b, x.gt, x.g, x.Ip, x.cu, coff, ckM, ckI, decay, order});
    const auto bit = [](bool on, int64_t b) { return on ? b : int64_t(0); };
    ctx->saved_data["scale"] = opt.scale;
    ctx->saved_data["bits"] = bit(opt.unc, NODE_UNC) | bit(opt.recurrent, NODE_RECURRENT) | bit(x.mu0.defined(), NODE_INIT) |
                              bit(opt.save_ckpt, NODE_CKPT) | bit(opt.carry_tc, NODE_CARRY_TC) | bit(x.cu.defined(), NODE_PACKED) |
                              bit(opt.segments > 1, NODE_CUT) | static_cast<int64_t>(x.q.scalar_type()) << NODE_IO_SHIFT;
    ctx->set_materialize_grads(false);
}

// The direct route's node: only what the caller gets back are outputs.
struct DirectFn : torch::autograd::Function<DirectFn> {
    static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b,
                                 const Tensor& gt, const Tensor& g, const Tensor& Ip, const Inputs& rest, const Options& opt) {
        Inputs x{q, k, v, b, gt, g, Ip, rest.mu0, rest.I0, rest.cu};
        FwdOut r = fwd_impl(x, opt);
        node_save(ctx, x, r.coff, r.order, r.ckM, r.ckI, r.decay, opt);
        variable_list out{r.o};
        if (opt.unc) out.push_back(r.o_var);
        if (opt.want_final) out.push_back(r.fmu), out.push_back(r.fI);
        return out;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) { return node_backward(ctx, grads, 9); }
};

// The registered operator's node: its eight outputs are what the schema names.
struct OpFn : torch::autograd::Function<OpFn> {
    static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b,
                                 const Tensor& gt, const Tensor& g, const Tensor& Ip, const Inputs& rest, const Options& opt) {
        at::AutoDispatchBelowADInplaceOrView below;
        auto o = [](const Tensor& t) { return t.defined() ? OptTensor(t) : std::nullopt; };
        auto [out, o_var, fmu, fI, ckM, ckI, coff, decay] =
            call_fwd_op(q, k, v, b, gt, g, Ip, o(rest.mu0), o(rest.I0), o(rest.cu), opt.scale, opt.unc, opt.save_ckpt,
                        opt.want_final, opt.recurrent, opt.segments);
        node_save(ctx, {q, k, v, b, gt, g, Ip, rest.mu0, rest.I0, rest.cu}, coff, Tensor(), ckM, ckI, decay, opt);
        return {out, o_var, fmu, fI, ckM, ckI, coff, decay};
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) { return node_backward(ctx, grads, 9); }
};
FwdTuple fwd_autograd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b, const Tensor& gt, const Tensor& g,
                      const Tensor& Ip, const OptTensor& init_mu, const OptTensor& init_I, const OptTensor& cu_seqlens,
                      double scale, bool uncertainty, bool save_ckpt, bool want_final, bool recurrent, int64_t num_segments) {
    Options opt;
    opt.scale = scale, opt.unc = uncertainty, opt.save_ckpt = save_ckpt, opt.want_final = want_final;
    opt.recurrent = recurrent, opt.segments = num_segments;
    if (num_segments > 1) opt.carry_tc = carry_switch();
    Inputs rest;
    rest.mu0 = init_mu.value_or(Tensor()), rest.I0 = init_I.value_or(Tensor()), rest.cu = cu_seqlens.value_or(Tensor());
    auto r = OpFn::apply(q, k, v, b, gt, g, Ip, rest, opt);
    return {r[0], r[1], r[2], r[3], r[4], r[5], r[6], r[7]};
}

// ---- decode ---------------------------------------------------------------------------------------------------
std::tuple<Tensor, Tensor> decode_impl(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b, const Tensor& gt,
                                       const Tensor& g, const Tensor& Ip, const Tensor& mu, const Tensor& I, double scale,
                                       bool unc) {
    const at::Device dev = q.device();
    check_inputs({q, k, v, b, gt, g, Ip, mu, I, Tensor()});
    TORCH_CHECK_VALUE(q.size(1) == 1, "decode_step takes exactly one token per sequence");
    c10::cuda::CUDAGuard guard(dev);
    const int64_t N = q.size(0), H = q.size(2), V = v.size(3);
    Tensor o = empty({N, 1, H, V}, q.scalar_type(), dev), o_var;
    if (unc) o_var = empty({N, 1, H, V}, q.scalar_type(), dev);
    palimpsa_fwd_params prm{};
    prm.struct_size = sizeof(prm);
    prm.p = make_problem(q, k, v, b, gt, g, Ip, Tensor(), Tensor(), Tensor(), mu, I, scale, unc ? PALIMPSA_FLAG_UNCERTAINTY : 0);
    prm.o = ptr(o), prm.o_var = ptr(o_var);
    prm.final_mu = ptr<float>(mu), prm.final_I = ptr<float>(I);
    check_rc(palimpsa_decode_step(&prm, stream_of(q)), "palimpsa decode step");
    return {o, o_var};
}
void bump_version(const Tensor& t) {
    if (!t.is_inference()) t.unsafeGetTensorImpl()->bump_version();
}
std::tuple<Tensor, Tensor> decode_cuda(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b, const Tensor& gt,
                                       const Tensor& g, const Tensor& Ip, const Tensor& mu_state, const Tensor& I_state,
                                       double scale, bool uncertainty) {
    auto [o, o_var] = decode_impl(dense(q), dense(k), dense(v), dense(b), dense(gt), dense(g), dense(Ip), mu_state, I_state,
                                  scale, uncertainty);
    return {o, o_var.defined() ? o_var : none_like(q, q.scalar_type())};
}
std::tuple<Tensor, Tensor> call_decode_op(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b, const Tensor& gt,
                                          const Tensor& g, const Tensor& Ip, const Tensor& mu, const Tensor& I, double scale,
                                          bool unc) {
    static auto op =
        c10::Dispatcher::singleton().findSchemaOrThrow("palimpsa_b200::decode_step", "").typed<decltype(decode_cuda)>();
    return op.call(q, k, v, b, gt, g, Ip, mu, I, scale, unc);
}
// The step is inference only: no graph, but the caches' version counters move, so that a saved use of them is noticed.
std::tuple<Tensor, Tensor> decode_autograd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b, const Tensor& gt,
                                           const Tensor& g, const Tensor& Ip, const Tensor& mu_state, const Tensor& I_state,
                                           double scale, bool uncertainty) {
    at::AutoDispatchBelowADInplaceOrView below;
    auto r = call_decode_op(q, k, v, b, gt, g, Ip, mu_state, I_state, scale, uncertainty);
    bump_version(mu_state);
    bump_version(I_state);
    return r;
}

std::tuple<Tensor, Tensor> decode_run(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& b_, const Tensor& gt_,
                                      const Tensor& g_, const Tensor& Ip_, const Tensor& mu, const Tensor& I,
                                      std::optional<double> scale, bool unc) {
    auto token = [&](const Tensor& t) { return q_.dim() == 3 ? t.unsqueeze(1) : t; };
    at::NoGradGuard no_grad;
    Tensor q = token(q_), k = token(k_), v = token(v_), b = token(b_), gt = token(gt_);
    TORCH_CHECK_VALUE(q.dim() == 4 && k.sizes() == q.sizes() && v.dim() == 4 && b.sizes() == v.sizes() &&
                          v.sizes().slice(0, 3) == q.sizes().slice(0, 3),
                      "expected q,k [N,1,H,K] and v,b [N,1,H,V]");
    const int64_t N = q.size(0), H = q.size(2), K = q.size(3), V = v.size(3);
    TORCH_CHECK_VALUE(q.size(1) == 1, "decode_step takes exactly one token per sequence");
    TORCH_CHECK_VALUE(gt.numel() == N * H && g_.numel() == H && Ip_.numel() == H, "expected gt [N,1,H] and g, Ip [H]");
    for (const Tensor* s : {&mu, &I})
        TORCH_CHECK_VALUE(s->scalar_type() == at::kFloat && s->is_contiguous() && s->sizes() == at::IntArrayRef({N, H, V, K}),
                          "state cache tensors must be contiguous float32 of shape (", N, ", ", H, ", ", V, ", ", K, ")");
    const at::ScalarType io = q.scalar_type();
    io_code(io);
    const double sc = scale ? *scale : 1.0 / std::sqrt((double)K);
    RECORD_FUNCTION("palimpsa_b200::decode_step", c10::ArrayRef<const c10::IValue>{});
    auto r = decode_impl(as(q, io), as(k, io), as(v, io), as(b, io), as(gt, at::kFloat), as(g_, at::kFloat), as(Ip_, at::kFloat),
                         mu, I, sc, unc);
    bump_version(mu);
    bump_version(I);
    return r;
}
// The entries Python calls give the interpreter lock back while they work: an allocation or a launch may wait for the
// device, and other threads have to be able to feed it meanwhile.
py::object decode_step(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b, const Tensor& gt, const Tensor& g,
                       const Tensor& Ip, const Tensor& mu, const Tensor& I, std::optional<double> scale, bool unc) {
    if (!plain({&q, &k, &v, &b, &gt, &g, &Ip, &mu, &I})) return not_plain();
    std::tuple<Tensor, Tensor> r;
    {
        py::gil_scoped_release no_gil;
        r = decode_run(q, k, v, b, gt, g, Ip, mu, I, scale, unc);
    }
    if (unc) return py::cast(r);
    return py::cast(std::get<0>(r));
}

// The token inputs of a replayed step into the graph's static buffers: one launch for those that are plain copies (same
// dtype, contiguous), tensor copies for the rest.
void copy_inputs(const std::vector<Tensor>& dst, const std::vector<OptTensor>& src) {
    const void* from[8];
    void* to[8];
    size_t bytes[8];
    int n = 0;
    c10::cuda::CUDAGuard guard(dst[0].device());
    for (size_t i = 0; i < dst.size(); ++i) {
        if (!given(src[i])) continue;
        const Tensor &d = dst[i], &s = *src[i];
        TORCH_CHECK_VALUE(s.numel() == d.numel(), "decode input ", i, ": ", s.numel(), " elements, expected ", d.numel());
        if (n < 8 && s.device() == d.device() && s.scalar_type() == d.scalar_type() && s.is_contiguous() && plain({&s})) {
            from[n] = s.const_data_ptr(), to[n] = d.data_ptr(), bytes[n++] = (size_t)d.nbytes();
            bump_version(d);
        } else {
            at::NoGradGuard no_grad;
            d.copy_(s.reshape(d.sizes()), /*non_blocking=*/true);
        }
    }
    check_rc(palimpsa_copy_buffers(from, to, bytes, n, stream_of(dst[0])), "decode inputs");
}

// ---- chunk_palimpsa / fused_recurrent_palimpsa ------------------------------------------------------------------
struct RunOut {
    Tensor o, o_var, fmu, fI;  // undefined where not asked for
};
RunOut run_impl(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b, const Tensor& gt, const Tensor& g,
                const Tensor& Ip, const OptTensor& mu0, const OptTensor& I0, std::optional<double> scale, bool want_final,
                bool unc, const OptTensor& cu, bool recurrent, std::optional<int64_t> num_segments, bool carry_tc) {
    if (given(cu)) {
        TORCH_CHECK_VALUE(q.size(0) == 1, recurrent ? "The batch size is expected to be 1 rather than " : "Batch size must be 1 for Varlen, got ",
                          q.size(0), recurrent ? " when using `cu_seqlens`." : "");
        TORCH_CHECK_VALUE(!recurrent || !given(mu0) || mu0->size(0) == cu->numel() - 1, "Initial states mismatch sequence length.");
    }
    TORCH_CHECK_VALUE(q.dim() == 4 && k.sizes() == q.sizes() && v.dim() == 4 && b.sizes() == v.sizes() &&
                          v.sizes().slice(0, 3) == q.sizes().slice(0, 3),
                      "expected q,k [B,T,H,K] and v,b [B,T,H,V]");
    const int64_t B = q.size(0), T = q.size(1), H = q.size(2), K = q.size(3), V = v.size(3);
    TORCH_CHECK_VALUE(gt.sizes() == at::IntArrayRef({B, T, H}) && g.sizes() == at::IntArrayRef({H}) && Ip.sizes() == at::IntArrayRef({H}),
                      "expected gt [B,T,H] and g, Ip [H]");
    Inputs x;
    x.cu = cu.value_or(Tensor()), x.mu0 = mu0.value_or(Tensor()), x.I0 = I0.value_or(Tensor());
    io_code(q.scalar_type());
    if (x.cu.defined()) x.cu = as(x.cu, at::kInt);
    const int64_t N = x.cu.defined() ? x.cu.numel() - 1 : B;
    TORCH_CHECK_VALUE(x.mu0.defined() == x.I0.defined(), "initial_mu_state and initial_I_state must be given together");
    if (x.mu0.defined()) {
        const std::array<int64_t, 4> dims{N, H, V, K};
        const at::IntArrayRef want(dims);
        TORCH_CHECK_VALUE(x.mu0.sizes() == want && x.I0.sizes() == want, "initial states must have shape (", N, ", ", H, ", ", V, ", ", K, ")");
        at::NoGradGuard no_grad;
        x.mu0 = as(x.mu0.requires_grad() ? x.mu0.detach() : x.mu0, at::kFloat);
        x.I0 = as(x.I0.requires_grad() ? x.I0.detach() : x.I0, at::kFloat);
    }
    // One io dtype per call: the widest of the four token tensors (the reference's kernels read each tensor in its own
    // dtype and compute in fp32, so a narrower choice would round an input the reference does not round; under autocast
    // its layers do pass fp32 q/k next to bf16 v).
    at::ScalarType io = q.scalar_type();
    for (const Tensor* t : {&k, &v, &b}) io = c10::promoteTypes(io, t->scalar_type());
    io_code(io);
    x.q = as(q, io), x.k = as(k, io), x.v = as(v, io), x.b = as(b, io);
    x.gt = as(gt, at::kFloat), x.g = as(g, at::kFloat), x.Ip = as(Ip, at::kFloat);
    Options opt;
    opt.scale = scale ? *scale : 1.0 / std::sqrt((double)K);
    opt.unc = unc, opt.want_final = want_final, opt.recurrent = recurrent, opt.carry_tc = carry_tc;
    if (at::GradMode::is_enabled())
        for (const Tensor* t : {&x.q, &x.k, &x.v, &x.b, &x.gt, &x.g, &x.Ip}) opt.save_ckpt |= t->requires_grad();
    opt.segments = num_segments ? *num_segments
                                : plan_segments(N, T, H, K, V, sm_count(q), opt.save_ckpt, io_code(io), unc, x.cu.defined());
    RECORD_FUNCTION("palimpsa_b200::fwd", c10::ArrayRef<const c10::IValue>{});  // as the operator is called in a profile
    Tensor o, o_var, fmu, fI;
    if (opt.save_ckpt) {
        auto r = DirectFn::apply(x.q, x.k, x.v, x.b, x.gt, x.g, x.Ip, x, opt);
        size_t i = 0;
        o = r[i++];
        if (unc) o_var = r[i++];
        if (want_final) fmu = r[i], fI = r[i + 1];
    } else {
        FwdOut r = fwd_impl(x, opt);
        o = r.o, o_var = r.o_var, fmu = r.fmu, fI = r.fI;
    }
    // o in q's dtype (the fused op: v's, with o_var in float32, as in the reference)
    const at::ScalarType o_dt = recurrent ? v.scalar_type() : q.scalar_type(), var_dt = recurrent ? at::kFloat : q.scalar_type();
    if (o.scalar_type() != o_dt) o = o.to(o_dt);
    if (unc && o_var.scalar_type() != var_dt) o_var = o_var.to(var_dt);
    return {o, o_var, fmu, fI};
}
py::object run(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b, const Tensor& gt, const Tensor& g,
               const Tensor& Ip, const OptTensor& mu0, const OptTensor& I0, std::optional<double> scale, bool want_final,
               bool unc, const OptTensor& cu, bool recurrent, std::optional<int64_t> num_segments, bool carry_tc) {
    const Tensor mu = mu0.value_or(Tensor()), I = I0.value_or(Tensor()), c = cu.value_or(Tensor());
    if (!plain({&q, &k, &v, &b, &gt, &g, &Ip, &mu, &I, &c})) return not_plain();
    RunOut r;
    {
        py::gil_scoped_release no_gil;
        r = run_impl(q, k, v, b, gt, g, Ip, mu0, I0, scale, want_final, unc, cu, recurrent, num_segments, carry_tc);
    }
    py::object out = unc ? py::cast(std::make_tuple(r.o, r.o_var)) : py::cast(r.o);
    if (want_final) return py::make_tuple(out, r.fmu, r.fI);
    return out;
}

// ---- the layer's element-wise sides (differentiable; palimpsa_b200/layers.py documents them) -----------------------
Tensor layer_workspace(int64_t tokens, int64_t H, int64_t V, const at::Device& dev) {
    return empty({std::max<int64_t>((int64_t)palimpsa_layer_workspace_bytes(tokens, (int32_t)H, (int32_t)V), 256)}, at::kByte, dev);
}
int64_t token_count(const Tensor& x) { return x.numel() ? x.numel() / (x.size(-1) * x.size(-2)) : 0; }
std::vector<int64_t> with_last(const Tensor& t, int64_t H, int64_t n) {  // [..., H, n] with t's leading dimensions
    auto s = t.sizes().vec();
    s[s.size() - 2] = H, s[s.size() - 1] = n;
    return s;
}
// The dtypes of the arguments as the caller passed them, a byte each (a value that hashes: see the operator's node).
int64_t pack_dtypes(std::initializer_list<at::ScalarType> ts) {
    int64_t bits = 0, shift = 0;
    for (at::ScalarType t : ts) bits |= static_cast<int64_t>(t) << shift, shift += 8;
    return bits;
}
at::ScalarType dtype_at(int64_t bits, size_t i) { return static_cast<at::ScalarType>(bits >> (8 * i) & 0xff); }
Tensor grad_in(const Tensor& g, at::IntArrayRef sizes, at::ScalarType dt, const at::Device& dev) {
    return g.defined() ? as(g, dt) : at::zeros(sizes, at::TensorOptions().dtype(dt).device(dev));
}

palimpsa_layer_prologue prologue_params(const std::vector<Tensor>& t) {
    palimpsa_layer_prologue a{};
    a.struct_size = sizeof(a);
    const Tensor &q = t[0], &x = t[2];
    a.io_dtype = io_code(x.scalar_type());
    a.H = (int)x.size(-2), a.Hq = (int)q.size(-2), a.K = (int)q.size(-1), a.V = (int)x.size(-1);
    a.tokens = token_count(x);
    a.q_raw = ptr(t[0]), a.k_raw = ptr(t[1]), a.x = ptr(t[2]), a.b_raw = ptr(t[3]), a.dt_raw = ptr(t[4]), a.bs_raw = ptr(t[5]);
    a.dt_bias = ptr<float>(t[6]), a.b_scale = ptr<float>(t[7]);
    return a;
}
struct PrologueFn : torch::autograd::Function<PrologueFn> {
    static variable_list forward(AutogradContext* ctx, const Tensor& q_raw, const Tensor& k_raw, const Tensor& x,
                                 const Tensor& b_raw, const Tensor& dt_raw, const Tensor& bs_raw, const Tensor& dt_bias,
                                 const Tensor& b_scale) {
        const at::ScalarType io = x.scalar_type();
        const at::Device dev = x.device();
        c10::cuda::CUDAGuard guard(dev);
        std::vector<Tensor> t;
        for (const Tensor* a : {&q_raw, &k_raw, &x, &b_raw, &dt_raw, &bs_raw, &dt_bias, &b_scale})
            t.push_back(as(*a, t.size() < 6 ? io : at::kFloat));
        const int64_t H = x.size(-2), K = q_raw.size(-1);
        const auto qs = with_last(x, H, K);
        Tensor q = empty(qs, io, dev), k = empty(qs, io, dev), v = empty(x.sizes(), io, dev), b = empty(x.sizes(), io, dev);
        Tensor gt = empty(x.sizes().slice(0, x.dim() - 1), at::kFloat, dev);
        palimpsa_layer_prologue a = prologue_params(t);
        a.q = ptr(q), a.k = ptr(k), a.v = ptr(v), a.b = ptr(b), a.gt = ptr<float>(gt);
        if (a.tokens > 0)  // an empty batch has nothing to launch (and no pointers)
            check_rc(palimpsa_layer_prologue_fwd(&a, stream_of(x)), "layer prologue");
        ctx->save_for_backward(t);
        ctx->saved_data["dtypes"] = pack_dtypes({q_raw.scalar_type(), k_raw.scalar_type(), io, b_raw.scalar_type(),
                                                 dt_raw.scalar_type(), bs_raw.scalar_type(), dt_bias.scalar_type(),
                                                 b_scale.scalar_type()});
        ctx->set_materialize_grads(false);
        return {q, k, v, b, gt};
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        auto t = ctx->get_saved_variables();
        const int64_t types = ctx->saved_data["dtypes"].toInt();
        const Tensor& x = t[2];
        const at::ScalarType io = x.scalar_type();
        const at::Device dev = x.device();
        c10::cuda::CUDAGuard guard(dev);
        const int64_t H = x.size(-2), V = x.size(-1);
        const auto qs = with_last(x, H, t[0].size(-1));
        const Tensor dq = grad_in(g[0], qs, io, dev), dk = grad_in(g[1], qs, io, dev), dv = grad_in(g[2], x.sizes(), io, dev),
                     db = grad_in(g[3], x.sizes(), io, dev), dgt = grad_in(g[4], t[4].sizes(), at::kFloat, dev);
        palimpsa_layer_prologue a = prologue_params(t);
        a.dq = ptr(dq), a.dk = ptr(dk), a.dv = ptr(dv), a.db = ptr(db), a.dgt = ptr<float>(dgt);
        variable_list out;
        for (int i = 0; i < 6; ++i) out.push_back(empty(t[i].sizes(), io, dev));
        for (int i = 0; i < 2; ++i) out.push_back(empty({H}, at::kFloat, dev));
        a.dq_raw = ptr(out[0]), a.dk_raw = ptr(out[1]), a.dx = ptr(out[2]), a.db_raw = ptr(out[3]), a.ddt_raw = ptr(out[4]);
        a.dbs_raw = ptr(out[5]), a.d_dt_bias = ptr<float>(out[6]), a.d_b_scale = ptr<float>(out[7]);
        Tensor ws = layer_workspace(a.tokens, H, V, dev);
        a.workspace = ptr(ws), a.workspace_bytes = (size_t)ws.numel();
        if (a.tokens > 0)
            check_rc(palimpsa_layer_prologue_bwd(&a, stream_of(x)), "layer prologue backward");
        else
            out[6].zero_(), out[7].zero_();
        for (size_t i = 0; i < out.size(); ++i)
            if (out[i].scalar_type() != dtype_at(types, i)) out[i] = out[i].to(dtype_at(types, i));
        for (int i : {6, 7})
            if (out[i].sizes() != t[i].sizes()) out[i] = out[i].view(t[i].sizes());
        return out;
    }
};
variable_list layer_prologue(const Tensor& q_raw, const Tensor& k_raw, const Tensor& x, const Tensor& b_raw, const Tensor& dt_raw,
                             const Tensor& bs_raw, const Tensor& dt_bias, const Tensor& b_scale) {
    require_cuda({&q_raw, &k_raw, &x, &b_raw, &dt_raw, &bs_raw, &dt_bias, &b_scale});
    io_code(x.scalar_type());
    const int64_t H = x.size(-2), Hq = q_raw.size(-2);
    TORCH_CHECK_VALUE(Hq > 0 && H % Hq == 0 && q_raw.sizes() == k_raw.sizes() && b_raw.sizes() == x.sizes() &&
                          q_raw.sizes().slice(0, q_raw.dim() - 2) == x.sizes().slice(0, x.dim() - 2),
                      "layer_prologue: q_raw/k_raw [...,Hq,K], x/b_raw [...,H,V] with H a multiple of Hq");
    const auto rows = x.sizes().slice(0, x.dim() - 1);
    TORCH_CHECK_VALUE(dt_raw.sizes() == rows && bs_raw.sizes() == rows && dt_bias.numel() == H && b_scale.numel() == H,
                      "layer_prologue: dt_raw/bs_raw [...,H], dt_bias/b_scale [H]");
    return PrologueFn::apply(q_raw, k_raw, x, b_raw, dt_raw, bs_raw, dt_bias, b_scale);
}

palimpsa_layer_epilogue epilogue_params(const std::vector<Tensor>& t, double eps, bool res, bool gated) {  // o, x, D, weight, gate
    palimpsa_layer_epilogue a{};
    a.struct_size = sizeof(a);
    a.io_dtype = io_code(t[0].scalar_type());
    a.H = (int)t[0].size(-2), a.V = (int)t[0].size(-1);
    a.flags = (res ? PALIMPSA_LAYER_RESIDUAL : 0) | (gated ? PALIMPSA_LAYER_GATE : 0);
    a.eps = (float)eps;
    a.tokens = token_count(t[0]);
    a.o = ptr(t[0]), a.x = ptr(t[1]), a.D = ptr<float>(t[2]), a.weight = ptr<float>(t[3]), a.gate = ptr(t[4]);
    return a;
}
struct EpilogueFn : torch::autograd::Function<EpilogueFn> {
    static variable_list forward(AutogradContext* ctx, const Tensor& o, const OptTensor& x, const OptTensor& D,
                                 const Tensor& weight, const OptTensor& gate, double eps) {
        const at::ScalarType io = o.scalar_type();
        c10::cuda::CUDAGuard guard(o.device());
        std::vector<Tensor> t{as(o, io), as_opt(x, io), as_opt(D, at::kFloat), as(weight, at::kFloat), as_opt(gate, io)};
        Tensor y = empty(o.sizes(), io, o.device());
        palimpsa_layer_epilogue a = epilogue_params(t, eps, given(x), given(gate));
        a.y = ptr(y);
        if (a.tokens > 0) check_rc(palimpsa_layer_epilogue_fwd(&a, stream_of(o)), "layer epilogue");
        ctx->save_for_backward(t);
        ctx->saved_data["dtypes"] = pack_dtypes({io, given(x) ? x->scalar_type() : io, given(D) ? D->scalar_type() : at::kFloat,
                                                 weight.scalar_type(), given(gate) ? gate->scalar_type() : io});
        ctx->saved_data["eps"] = eps;
        ctx->saved_data["parts"] = static_cast<int64_t>((given(x) ? 1 : 0) | (given(gate) ? 2 : 0));
        return {y};
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        auto t = ctx->get_saved_variables();
        const int64_t types = ctx->saved_data["dtypes"].toInt(), parts = ctx->saved_data["parts"].toInt();
        const bool res = (parts & 1) != 0, gated = (parts & 2) != 0;
        const Tensor& o = t[0];
        const at::ScalarType io = o.scalar_type();
        const at::Device dev = o.device();
        c10::cuda::CUDAGuard guard(dev);
        const int64_t H = o.size(-2), V = o.size(-1);
        const Tensor dy = grad_in(g[0], o.sizes(), io, dev);
        Tensor d_o = empty(o.sizes(), io, dev), dx, dD, dw = empty({V}, at::kFloat, dev), dgate;
        if (res) dx = empty(o.sizes(), io, dev), dD = empty({H}, at::kFloat, dev);
        if (gated) dgate = empty(o.sizes(), io, dev);
        palimpsa_layer_epilogue a = epilogue_params(t, ctx->saved_data["eps"].toDouble(), res, gated);
        a.dy = ptr(dy), a.d_o = ptr(d_o), a.dx = ptr(dx), a.dgate = ptr(dgate), a.dD = ptr<float>(dD), a.dweight = ptr<float>(dw);
        Tensor ws = layer_workspace(a.tokens, H, V, dev);
        a.workspace = ptr(ws), a.workspace_bytes = (size_t)ws.numel();
        if (a.tokens > 0) {
            check_rc(palimpsa_layer_epilogue_bwd(&a, stream_of(o)), "layer epilogue backward");
        } else {
            dw.zero_();
            if (dD.defined()) dD.zero_();
        }
        variable_list out{d_o, dx, dD, dw, dgate, Tensor()};
        for (size_t i = 0; i < 5; ++i)
            if (out[i].defined() && out[i].scalar_type() != dtype_at(types, i)) out[i] = out[i].to(dtype_at(types, i));
        for (int i : {2, 3})
            if (out[i].defined() && out[i].sizes() != t[i].sizes()) out[i] = out[i].view(t[i].sizes());
        return out;
    }
};
Tensor layer_epilogue(const Tensor& o, const OptTensor& x, const OptTensor& D, const Tensor& weight, const OptTensor& gate,
                      double eps) {
    const Tensor x_ = x.value_or(Tensor()), D_ = D.value_or(Tensor()), g_ = gate.value_or(Tensor());
    require_cuda({&o, &x_, &D_, &weight, &g_});
    io_code(o.scalar_type());
    TORCH_CHECK_VALUE(given(x) == given(D), "layer_epilogue: pass both x and D (residual) or neither");
    TORCH_CHECK_VALUE(!given(x) || (x->sizes() == o.sizes() && D->numel() == o.size(-2)), "layer_epilogue: x like o, D [H]");
    TORCH_CHECK_VALUE(!given(gate) || gate->sizes() == o.sizes(), "layer_epilogue: gate like o");
    TORCH_CHECK_VALUE(weight.numel() == o.size(-1), "layer_epilogue: weight [V]");
    return EpilogueFn::apply(o, x, D, weight, gate, eps)[0];
}

int64_t plan_segments_py(int64_t N, int64_t T, int64_t H, int64_t K, int64_t V, int64_t sms, bool backward, int64_t io, bool unc,
                         bool packed) {
    return plan_segments(N, T, H, K, V, sms, backward, (int)io, unc, packed);
}

}  // namespace

TORCH_LIBRARY(palimpsa_b200, m) {
    m.def("fwd(Tensor q, Tensor k, Tensor v, Tensor b, Tensor gt, Tensor g, Tensor Ip, Tensor? init_mu, Tensor? init_I, "
          "Tensor? cu_seqlens, float scale, bool uncertainty, bool save_ckpt, bool want_final, bool recurrent, "
          "int num_segments) -> (Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor)",
          {at::Tag::pt2_compliant_tag});
    m.def("bwd(Tensor do, Tensor? do_var, Tensor q, Tensor k, Tensor v, Tensor b, Tensor gt, Tensor g, Tensor Ip, "
          "Tensor? cu_seqlens, Tensor? chunk_offsets, Tensor ckpt_M, Tensor ckpt_I, float scale, bool explicit_init, "
          "bool recurrent, Tensor? seg_decay) -> (Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor)",
          {at::Tag::pt2_compliant_tag});
    m.def("decode_step(Tensor q, Tensor k, Tensor v, Tensor b, Tensor gt, Tensor g, Tensor Ip, Tensor(a!) mu_state, "
          "Tensor(b!) I_state, float scale, bool uncertainty) -> (Tensor, Tensor)",
          {at::Tag::pt2_compliant_tag});
}
TORCH_LIBRARY_IMPL(palimpsa_b200, CUDA, m) {
    m.impl("fwd", fwd_cuda);
    m.impl("bwd", bwd_cuda);
    m.impl("decode_step", decode_cuda);
}
TORCH_LIBRARY_IMPL(palimpsa_b200, Autograd, m) {
    m.impl("fwd", fwd_autograd);
    m.impl("bwd", torch::autograd::autogradNotImplementedFallback());
    m.impl("decode_step", decode_autograd);
}

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.def("run", &run);
    m.def("decode_step", &decode_step);
    m.def("copy_inputs", &copy_inputs, py::call_guard<py::gil_scoped_release>());
    m.def("layer_prologue", &layer_prologue, py::call_guard<py::gil_scoped_release>());
    m.def("layer_epilogue", &layer_epilogue, py::call_guard<py::gil_scoped_release>());
    m.def("plan_segments", &plan_segments_py);
    m.def("abi_version", [] { return PALIMPSA_ABI_VERSION; });
}
