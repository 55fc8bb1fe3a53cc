// Host side of the Python operators: argument checks, allocation of results, the autograd nodes and the calls
// into the C ABI, in native code.  One call costs the host a few microseconds; the same steps in Python
// (ctypes conversions, a Python autograd.Function, tensors created one by one) cost 35-60 us per direction, more than the
// kernels of small problems and of a decode step take.
//
// PyTorch supplies device memory, streams and the autograd graph only; all arithmetic is in libdsqg_b200.so.
#include <torch/extension.h>

#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/Exceptions.h>

#include <cublasLt.h>
#include <cublas_v2.h>

#include <array>
#include <cmath>
#include <map>
#include <memory>
#include <mutex>
#include <optional>
#include <sstream>

#include "dsqg_b200.h"

namespace py = pybind11;
using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

namespace {

// An offset set, converted once and kept for the life of the process (programs use a handful): autograd nodes and
// the Python cache (ops._offsets) hold plain pointers to it.
struct Offsets {
    std::vector<int32_t> v;
    int J() const { return (int)v.size(); }
};

const Offsets* intern_offsets(const std::vector<int32_t>& v) {
    static std::mutex mu;
    static std::map<std::vector<int32_t>, std::unique_ptr<Offsets>> table;
    std::lock_guard<std::mutex> lock(mu);
    std::unique_ptr<Offsets>& o = table[v];
    if (!o) { o = std::make_unique<Offsets>(); o->v = v; }
    return o.get();
}

// Raises dwarf_b200.DSQGError for a non-zero status.
void check(int status, const char* where) {
    if (status == DSQG_OK) return;
    py::gil_scoped_acquire gil;
    py::module_::import("dwarf_b200._lib").attr("check")(status, where);
    throw std::runtime_error(std::string(where) + " failed");
}

// Runs the body of a backward node: the autograd engine's threads carry Python errors in its own exception type, and start
// without a CUDA context, which cuBLAS would remark on.
template <typename F> auto backward_body(const Tensor& on, F f) {
    static thread_local int ready = -1;
    if (on.defined() && on.is_cuda() && ready != on.device().index()) {
        ready = on.device().index();
        const int before = c10::cuda::current_device();
        c10::cuda::SetDevice(ready, /*force=*/true);
        c10::cuda::SetDevice(before);
    }
    try {
        return f();
    } catch (py::error_already_set& e) {
        py::gil_scoped_acquire gil;
        e.restore();
        python_error err;
        err.persist();
        throw err;
    }
}

int dtype_code(const Tensor& t) {
    if (t.scalar_type() == at::kBFloat16) return DSQG_DTYPE_BF16;
    if (t.scalar_type() == at::kFloat) return DSQG_DTYPE_F32;
    throw py::type_error(std::string("dsqg: q/k/v must be bfloat16 or float32, got ") + toString(t.scalar_type()));
}

std::string shape_of(const Tensor& t) {
    std::ostringstream s;
    s << t.sizes();
    return s.str();
}

void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
float* fptr(const Tensor& t) { return t.defined() ? static_cast<float*>(t.data_ptr()) : nullptr; }
void* stream_of(const Tensor& t) { return at::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// Uninitialised device tensors straight from the allocator: a dispatched at::empty costs 2.6 us on an autograd thread, this
// one less than a third, and a backward call makes six.
Tensor new_tensor(at::IntArrayRef sizes, at::ScalarType dt, const Tensor& on) { return at::detail::empty_cuda(sizes, dt, on.device(), std::nullopt); }
Tensor new_like(const Tensor& t) { return t.defined() ? new_tensor(t.sizes(), t.scalar_type(), t) : t; }

// A parameter as the kernels read it: fp32 and contiguous (no copy where it is so already; it may be the caller's own tensor).
Tensor f32c(const Tensor& t) {
    if (!t.defined() || (t.scalar_type() == at::kFloat && t.is_contiguous())) return t;
    return t.detach().to(at::kFloat).contiguous();
}
// The kernels around the GEMMs and the GEMM plans want 16-byte pointers; a parameter that is a view of a flat buffer, or a caller's
// activation, may start anywhere and is copied then.
bool on_16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
Tensor aligned(const Tensor& t) { return !t.defined() || on_16(t.data_ptr()) ? t : t.detach().clone(); }
Tensor like_param(Tensor g, at::ScalarType dt) { return g.defined() && g.scalar_type() != dt ? g.to(dt) : g; }
Tensor opt(const std::optional<Tensor>& t) { return t.has_value() ? *t : Tensor(); }
at::ScalarType type_of(const Tensor& t) { return t.defined() ? t.scalar_type() : at::kFloat; }

bool shape_is(const Tensor& t, std::initializer_list<int64_t> s) { return t.sizes() == at::IntArrayRef(s); }

// The kernels get plain pointers: a tensor on the host or on another GPU would be read as if it were on this one.
void check_device(const char* who, const Tensor& on, std::initializer_list<const Tensor*> ts) {
    for (const Tensor* t : ts)
        if (t->defined() && t->device() != on.device()) throw py::value_error(std::string(who) + ": all tensors must be on " + on.device().str() + ", got one on " + t->device().str());
}

void check_inputs(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& pb, const Tensor& hg, const Tensor& se, int J) {
    if (!q.is_cuda()) throw std::runtime_error("dsqg: tensors must live on a CUDA device (there is no CPU path)");
    if (q.dim() != 4) throw py::value_error("dsqg: q must be [B,H,N,HD], got " + shape_of(q));
    const int64_t H = q.size(1), D = q.size(3);
    for (const Tensor* t : {&k, &v})
        if (t->sizes() != q.sizes() || t->scalar_type() != q.scalar_type() || t->device() != q.device())
            throw py::value_error(std::string("dsqg: ") + (t == &k ? "k" : "v") + " must match q in shape, dtype and device");
    auto want = [](const char* n, int64_t a, int64_t b, const Tensor& t) {
        throw py::value_error(std::string("dsqg: ") + n + " must be [" + std::to_string(a) + (b ? "," + std::to_string(b) : "") + "], got " + shape_of(t));
    };
    if (!shape_is(pb, {J, H})) want("pos_bias", J, H, pb);
    if (se.defined() && !shape_is(se, {J, D})) want("scale_embed", J, D, se);
    if (hg.defined() && !shape_is(hg, {H})) want("head_gain", H, 0, hg);
    check_device("dsqg", q, {&pb, &se, &hg});
}

// Head dimension the kernels are called with.  The bf16 tensor-core kernels exist for multiples of 32 up to 128; another bf16 width
// is zero-padded up to the next of those where they take the padded problem, with the scale 1/sqrt(D) of the true width:
// several times faster than the CUDA-core kernels on the odd width (the reference pads to a power of two inside its kernels,
// kernels/dsqg_attention_v2.py:344).  The widths 48 and 80 (the reference's 85M condM model, train/train_2048_85m_condM.py:67-69) have
// kernels of their own for the usual dense window without scale_embed (B8 H8 N2048 HD80 forward + backward: the copies into
// 96 columns and back took 232 us of 454).  fp32 is never padded.
int64_t padded_head_dim(int64_t D, bool bf16, const Offsets& off, bool has_se) {
    if (!bf16 || D % 32 == 0 || D > 128 || D % 8 != 0) return D;
    const int64_t Dp = (D + 31) / 32 * 32;
    const bool own = (D == 48 || D == 80) && !has_se;
    if (own && dsqg_tensor_core_path(DSQG_DTYPE_BF16, 96, off.v.data(), off.J(), 0)) return D;
    return dsqg_tensor_core_path(DSQG_DTYPE_BF16, (int)Dp, off.v.data(), off.J(), has_se) ? Dp : D;
}

Tensor pad_to(const Tensor& t, int64_t Dp) { return t.defined() ? at::constant_pad_nd(t, {0, Dp - t.size(-1)}) : t; }

// Scratch for one backward call, returned to the caching allocator when it leaves scope.
at::DataPtr scratch_for(size_t bytes) { return c10::cuda::CUDACachingAllocator::get()->allocate(bytes); }

// ------------------------------------------------------------------------------------ dsqg_attention
struct Forward { Tensor q, k, v, pb, hg, se, out, lse; int64_t D; };

Forward attention_forward(const Tensor& q0, const Tensor& k0, const Tensor& v0, const Tensor& pos_bias, const Tensor& head_gain,
                          const Tensor& scale_embed, const Offsets& off) {
    check_inputs(q0, k0, v0, pos_bias, head_gain, scale_embed, off.J());
    const int dt = dtype_code(q0);
    const c10::cuda::CUDAGuard guard(q0.device());
    Forward f;
    f.pb = f32c(pos_bias); f.hg = f32c(head_gain); f.se = f32c(scale_embed);
    f.D = q0.size(3);
    const int64_t Dp = padded_head_dim(f.D, dt == DSQG_DTYPE_BF16, off, scale_embed.defined());
    f.q = q0; f.k = k0; f.v = v0;
    if (Dp != f.D) {                                    // zero columns change no score and give zero outputs
        f.q = pad_to(f.q, Dp); f.k = pad_to(f.k, Dp); f.v = pad_to(f.v, Dp); f.se = pad_to(f.se, Dp);
    }
    f.q = f.q.contiguous(); f.k = f.k.contiguous(); f.v = f.v.contiguous();
    const int64_t B = f.q.size(0), H = f.q.size(1), N = f.q.size(2);
    f.out = new_like(f.q);
    f.lse = new_tensor({B, H, N}, at::kFloat, f.q);
    check(dsqg_fwd_scaled(ptr(f.q), ptr(f.k), ptr(f.v), fptr(f.pb), fptr(f.se), fptr(f.hg), off.v.data(), off.J(), ptr(f.out), fptr(f.lse),
                          (int)B, (int)H, (int)N, (int)Dp, dt, stream_of(f.q), (float)(1.0 / std::sqrt((double)f.D))), "dsqg_fwd");
    return f;
}

Tensor narrow_cols(const Tensor& t, int64_t D) { return t.defined() && t.size(-1) != D ? t.narrow(-1, 0, D).contiguous() : t; }

std::vector<int64_t> types_of(const Tensor& a, const Tensor& b, const Tensor& c) {
    return {(int64_t)type_of(a), (int64_t)type_of(b), (int64_t)type_of(c)};
}
at::ScalarType type_at(AutogradContext* ctx, int i) { return (at::ScalarType)ctx->saved_data["types"].toIntVector()[i]; }
const Offsets& offsets_of(AutogradContext* ctx) { return *reinterpret_cast<const Offsets*>((intptr_t)ctx->saved_data["offsets"].toInt()); }

// Saves q, k, v, pos_bias, head_gain, scale_embed, out, lse like the reference (kernels/dsqg_attention_v3.py:384).
struct AttentionNode : torch::autograd::Function<AttentionNode> {
    static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& pos_bias,
                          const std::optional<Tensor>& hg, const std::optional<Tensor>& se, const Offsets* off) {
        const Tensor head_gain = opt(hg), scale_embed = opt(se);
        Forward f = attention_forward(q, k, v, pos_bias, head_gain, scale_embed, *off);
        ctx->save_for_backward({f.q, f.k, f.v, f.pb, f.hg, f.se, f.out, f.lse});
        ctx->saved_data["offsets"] = (int64_t)(intptr_t)off;
        ctx->saved_data["D"] = f.D;
        ctx->saved_data["types"] = types_of(pos_bias, head_gain, scale_embed);
        return narrow_cols(f.out, f.D);
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        return backward_body(grads[0], [&] { return run(ctx, grads[0]); });
    }

    static variable_list run(AutogradContext* ctx, Tensor dout) {
        const variable_list s = ctx->get_saved_variables();
        const Tensor &q = s[0], &k = s[1], &v = s[2], &pb = s[3], &hg = s[4], &se = s[5], &out = s[6], &lse = s[7];
        const Offsets& off = offsets_of(ctx);
        const int64_t D = ctx->saved_data["D"].toInt(), B = q.size(0), H = q.size(1), N = q.size(2), Dp = q.size(3);
        const c10::cuda::CUDAGuard guard(q.device());
        if (dout.scalar_type() != q.scalar_type()) dout = dout.to(q.scalar_type());
        if (Dp != D) dout = pad_to(dout, Dp);
        dout = dout.contiguous();                                  // kernels/dsqg_attention_v3.py:394
        Tensor dq = new_like(q), dk = new_like(k), dv = new_like(v), dpb = new_like(pb);
        Tensor dhg = new_like(hg), dse = new_like(se);
        const size_t bytes = dsqg_bwd_scratch_bytes(off.J(), (int)B, (int)H, (int)N, (int)Dp, se.defined());
        const at::DataPtr scratch = scratch_for(bytes);
        check(dsqg_bwd_scaled(ptr(q), ptr(k), ptr(v), fptr(pb), fptr(se), fptr(hg), off.v.data(), off.J(), ptr(out), fptr(lse), ptr(dout),
                              ptr(dq), ptr(dk), ptr(dv), fptr(dpb), fptr(dse), fptr(dhg), scratch.get(), bytes,
                              (int)B, (int)H, (int)N, (int)Dp, dtype_code(q), stream_of(q), (float)(1.0 / std::sqrt((double)D))), "dsqg_bwd");
        return {narrow_cols(dq, D), narrow_cols(dk, D), narrow_cols(dv, D), like_param(dpb, type_at(ctx, 0)),
                like_param(dhg, type_at(ctx, 1)), like_param(narrow_cols(dse, D), type_at(ctx, 2)), Tensor()};
    }
};

bool wants_grad(std::initializer_list<const Tensor*> ts) {
    if (!at::GradMode::is_enabled()) return false;
    for (const Tensor* t : ts)
        if (t->defined() && t->requires_grad()) return true;
    return false;
}

Tensor attention(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& pb, const std::optional<Tensor>& hg,
                 const std::optional<Tensor>& se, const Offsets* off) {
    py::gil_scoped_release no_gil;
    const Tensor h = opt(hg), e = opt(se);
    if (wants_grad({&q, &k, &v, &pb, &h, &e})) return AttentionNode::apply(q, k, v, pb, hg, se, off);
    const Forward f = attention_forward(q, k, v, pb, h, e, *off);
    return narrow_cols(f.out, f.D);
}

std::tuple<Tensor, Tensor> forward_lse(const Tensor& q0, const Tensor& k0, const Tensor& v0, const Tensor& pb0, const std::optional<Tensor>& hg0,
                                       const std::optional<Tensor>& se0, const Offsets* off) {
    check_inputs(q0, k0, v0, pb0, opt(hg0), opt(se0), off->J());
    const int dt = dtype_code(q0);
    const c10::cuda::CUDAGuard guard(q0.device());
    const Tensor q = q0.contiguous(), k = k0.contiguous(), v = v0.contiguous(), pb = f32c(pb0), hg = f32c(opt(hg0)), se = f32c(opt(se0));
    Tensor out = new_like(q);
    Tensor lse = new_tensor({q.size(0), q.size(1), q.size(2)}, at::kFloat, q);
    check(dsqg_fwd(ptr(q), ptr(k), ptr(v), fptr(pb), fptr(se), fptr(hg), off->v.data(), off->J(), ptr(out), fptr(lse), (int)q.size(0),
                   (int)q.size(1), (int)q.size(2), (int)q.size(3), dt, stream_of(q)), "dsqg_fwd");
    return {out, lse};
}

// ------------------------------------------------------------------------------------ packed projection output
// What a packed forward leaves for its backward.  proj: the projection output [B*N, cols] (row-major) that q, k, v and, without a tensor of
// its own, the gate are read from in place; keep: the copies of q, k, v that stand in for it (dsqg_packed_keep_bytes).
struct PackedForward { Tensor proj, gate, pb, hg, se, y, lse, keep; };

// q, k, v at columns 0, H*D, 2*H*D of rows of `cols` elements; the gate at column 3*H*D of the same rows or in a tensor laid out like y.
dsqg_packed describe(const PackedForward& f, void* proj, int64_t cols, const Offsets& off) {
    const int64_t B = f.lse.size(0), H = f.lse.size(1), N = f.lse.size(2), D = f.y.size(2) / H;
    dsqg_packed p = {};
    char* at = static_cast<char*>(proj);
    p.q = at; p.k = at + H * D * 2; p.v = at + 2 * H * D * 2;
    p.qkv_strides = {N * cols, D, cols};
    p.out_strides = {N * H * D, D, H * D};
    p.gate = f.gate.defined() ? ptr(f.gate) : cols == 4 * H * D ? at + 3 * H * D * 2 : nullptr;
    p.gate_strides = f.gate.defined() ? p.out_strides : p.qkv_strides;
    p.pos_bias = fptr(f.pb); p.scale_embed = fptr(f.se); p.head_gain = fptr(f.hg);
    p.offsets = off.v.data(); p.J = off.J();
    p.B = (int)B; p.H = (int)H; p.N = (int)N; p.D = (int)D;
    p.out = ptr(f.y); p.lse = fptr(f.lse); p.keep = ptr(f.keep);
    return p;
}

// proj [.., cols]; with_grad: whether a backward will follow.
PackedForward packed_forward(const Tensor& proj, int64_t B, int64_t N, int64_t H, int64_t D, int64_t cols, const Tensor& gate, const Tensor& pos_bias,
                             const Tensor& head_gain, const Tensor& scale_embed, const Offsets& off, bool with_grad) {
    const int64_t J = off.J();
    check_device("dsqg", proj, {&gate, &pos_bias, &head_gain, &scale_embed});
    PackedForward f;
    f.proj = proj;
    f.gate = gate.defined() ? gate.contiguous() : gate;
    f.pb = f32c(pos_bias); f.hg = f32c(head_gain); f.se = f32c(scale_embed);
    if (!shape_is(f.pb, {J, H})) throw py::value_error("dsqg: pos_bias must be [" + std::to_string(J) + "," + std::to_string(H) + "], got " + shape_of(f.pb));
    if (f.se.defined() && !shape_is(f.se, {J, D}))
        throw py::value_error("dsqg: scale_embed must be [" + std::to_string(J) + "," + std::to_string(D) + "], got " + shape_of(f.se));
    f.y = new_tensor({B, N, H * D}, at::kBFloat16, proj);
    f.lse = new_tensor({B, H, N}, at::kFloat, proj);
    // a gated backward has dout in contiguous rows of its own; without a gate dy stays where it is and the copies would gain less than they cost
    const bool gated = f.gate.defined() || cols == 4 * H * D;
    if (with_grad && gated && dsqg_packed_keep_bytes((int)B, (int)H, (int)N, (int)D)) f.keep = new_tensor({3, B, H, N, D}, at::kBFloat16, proj);
    const dsqg_packed p = describe(f, ptr(proj), cols, off);
    check(dsqg_packed_fwd(&p, stream_of(proj)), "dsqg_packed_fwd");
    return f;
}

struct PackedGrads { Tensor dproj, dgate, dpb, dhg, dse; };

// dproj [B*N, cols], the gate's gradient in the last quarter of 4*H*D columns or in a tensor of its own; proj may be undefined where
// keep stands in for it and the gate has a tensor of its own.
PackedGrads packed_backward(const PackedForward& f, const Tensor& dy, int64_t cols, const Offsets& off) {
    const int64_t B = f.lse.size(0), N = f.lse.size(2);
    PackedGrads g;
    g.dproj = new_tensor({B * N, cols}, at::kBFloat16, dy);
    if (cols == 3 * f.y.size(2)) g.dgate = new_like(f.gate);
    g.dpb = new_like(f.pb); g.dhg = new_like(f.hg); g.dse = new_like(f.se);
    const dsqg_packed p = describe(f, f.proj.defined() ? ptr(f.proj) : ptr(f.keep), cols, off);
    const int64_t third = (int64_t)p.H * p.D * 2;
    char* at = static_cast<char*>(ptr(g.dproj));
    dsqg_packed_grads d = {};
    d.dy = ptr(dy); d.dq = at; d.dk = at + third; d.dv = at + 2 * third;
    d.dgate = g.dgate.defined() ? ptr(g.dgate) : at + 3 * third;
    d.dpos_bias = fptr(g.dpb); d.dscale_embed = fptr(g.dse); d.dhead_gain = fptr(g.dhg);
    const size_t bytes = dsqg_packed_bwd_scratch_bytes(&p);
    const at::DataPtr scratch = scratch_for(bytes);
    check(dsqg_packed_bwd_gate(&p, &d, g.dgate.defined() ? &p.gate_strides : &p.qkv_strides, scratch.get(), bytes, stream_of(dy)), "dsqg_packed_bwd");
    return g;
}

PackedForward packed_op(const Tensor& qkv, const Tensor& gate, const Tensor& pos_bias, const Tensor& head_gain, const Tensor& scale_embed,
                        const Offsets& off, bool with_grad) {
    if (qkv.dim() != 5 || qkv.size(2) != 3 || qkv.scalar_type() != at::kBFloat16 || !qkv.is_contiguous())
        throw py::value_error("dsqg packed: qkv must be a contiguous bf16 [B,N,3,H,HD] tensor");
    const int64_t B = qkv.size(0), N = qkv.size(1), H = qkv.size(3), D = qkv.size(4);
    if (gate.defined() && (gate.scalar_type() != at::kBFloat16 || !shape_is(gate, {B, N, H * D})))
        throw py::value_error("dsqg packed: gate must be bf16 [B,N,H*HD]");
    if (!qkv.is_cuda()) throw std::runtime_error("dsqg: tensors must live on a CUDA device (there is no CPU path)");
    const c10::cuda::CUDAGuard guard(qkv.device());
    return packed_forward(qkv, B, N, H, D, 3 * H * D, gate, pos_bias, head_gain, scale_embed, off, with_grad);
}

Tensor bf16c(const Tensor& t) { return (t.scalar_type() == at::kBFloat16 ? t : t.to(at::kBFloat16)).contiguous(); }

struct PackedNode : torch::autograd::Function<PackedNode> {
    static Tensor forward(AutogradContext* ctx, const Tensor& qkv, const std::optional<Tensor>& gate, const Tensor& pos_bias,
                          const std::optional<Tensor>& hg, const std::optional<Tensor>& se, const Offsets* off) {
        const Tensor head_gain = opt(hg), scale_embed = opt(se);
        PackedForward f = packed_op(qkv, opt(gate), pos_bias, head_gain, scale_embed, *off, true);
        ctx->save_for_backward({f.keep.defined() ? Tensor() : qkv, f.gate, f.pb, f.hg, f.se, f.y, f.lse, f.keep});
        ctx->saved_data["offsets"] = (int64_t)(intptr_t)off;
        ctx->saved_data["types"] = types_of(pos_bias, head_gain, scale_embed);
        return f.y;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        return backward_body(grads[0], [&] { return run(ctx, grads[0]); });
    }
    static variable_list run(AutogradContext* ctx, const Tensor& dy) {
        const variable_list s = ctx->get_saved_variables();
        const PackedForward f = {s[0], s[1], s[2], s[3], s[4], s[5], s[6], s[7]};
        const c10::cuda::CUDAGuard guard(dy.device());
        const int64_t B = f.lse.size(0), H = f.lse.size(1), N = f.lse.size(2), D = f.y.size(2) / H;
        const PackedGrads g = packed_backward(f, bf16c(dy), 3 * H * D, offsets_of(ctx));
        return {g.dproj.view({B, N, 3, H, D}), g.dgate, like_param(g.dpb, type_at(ctx, 0)), like_param(g.dhg, type_at(ctx, 1)),
                like_param(g.dse, type_at(ctx, 2)), Tensor()};
    }
};

Tensor attention_packed(const Tensor& qkv, const std::optional<Tensor>& gate, const Tensor& pb, const std::optional<Tensor>& hg,
                        const std::optional<Tensor>& se, const Offsets* off) {
    py::gil_scoped_release no_gil;
    const Tensor g = opt(gate), h = opt(hg), e = opt(se);
    if (wants_grad({&qkv, &g, &pb, &h, &e})) return PackedNode::apply(qkv, gate, pb, hg, se, off);
    return packed_op(qkv, g, pb, h, e, *off, false).y;
}

// ------------------------------------------------------------------------------------ causal mean
Tensor causal_mean_run(const Tensor& x, bool reverse) {
    const c10::cuda::CUDAGuard guard(x.device());
    Tensor out = new_like(x);
    check(dsqg_causal_mean(ptr(x), ptr(out), (int)x.size(0), (int)x.size(1), (int)x.size(2), dtype_code(x), reverse, stream_of(x)), "dsqg_causal_mean");
    return out;
}
struct CausalMeanNode : torch::autograd::Function<CausalMeanNode> {
    static Tensor forward(AutogradContext*, const Tensor& x) { return causal_mean_run(x, false); }
    static variable_list backward(AutogradContext*, variable_list grads) {
        return backward_body(grads[0], [&] { return variable_list{causal_mean_run(grads[0].contiguous(), true)}; });
    }
};
Tensor causal_mean(const Tensor& x0) {
    py::gil_scoped_release no_gil;
    if (!x0.is_cuda() || x0.dim() != 3 || (x0.scalar_type() != at::kBFloat16 && x0.scalar_type() != at::kFloat))
        throw py::value_error("causal_mean: x must be a CUDA [B,N,D] tensor in bfloat16 or float32");
    const Tensor x = x0.contiguous();
    return wants_grad({&x}) ? CausalMeanNode::apply(x) : causal_mean_run(x, false);
}

// ------------------------------------------------------------------------------------ whole layers under bf16 autocast
// The attention layer and the interference block as one autograd node each: what PyTorch runs as some ninety launches a
// step (1.9 ms of host time for 0.95 ms of GPU work at B8 N2048 dim 256) is their GEMMs (cuBLAS through ATen), the operator
// and the kernels of csrc/dsqg_layer.cu.  Weight gradients leave the GEMM in fp32 instead of being rounded to bf16 and cast.

// Autocast and autograd are done by hand inside the nodes.
struct NoAutocast {
    c10::impl::ExcludeDispatchKeyGuard guard{c10::autocast_dispatch_keyset};
    at::AutoDispatchBelowADInplaceOrView below;
};

// Row-major C[M,N] = op(A) . op(B) (+ bias[N]) on bf16 operands, C in bf16 or fp32, through cuBLASLt with plans kept per thread and
// problem: a call costs the host 4 us where at::linear and at::mm (dispatch, checks, a heuristic query each time) take 16-22, and
// a layer's step makes eleven.
struct GemmPlan {
    cublasLtMatmulDesc_t op = nullptr;
    cublasLtMatrixLayout_t a = nullptr, b = nullptr, c = nullptr;
    cublasLtMatmulAlgo_t algo;
    size_t workspace = 0;
    GemmPlan() = default;
    GemmPlan(const GemmPlan&) = delete;
    ~GemmPlan() {
        if (a) cublasLtMatrixLayoutDestroy(a);
        if (b) cublasLtMatrixLayoutDestroy(b);
        if (c) cublasLtMatrixLayoutDestroy(c);
        if (op) cublasLtMatmulDescDestroy(op);
    }
};
void lt_check(cublasStatus_t s, const char* what) {
    if (s != CUBLAS_STATUS_SUCCESS) throw std::runtime_error(std::string("dsqg: ") + what + ": " + cublasGetStatusString(s));
}
using GemmKey = std::array<int64_t, 9>;       // device, M, N, K, transposes and bias, output type, workspace, lda, reduction schemes

// The ways a plan may split its contraction, by torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction (as nn.Linear
// has it): partial sums in the output's 16 bits, in fp32 only, or no split at all.
uint32_t reduction_schemes() {
    switch (at::globalContext().allowBF16ReductionCuBLAS()) {
        case at::CuBLASReductionOption::AllowReducedPrecisionWithSplitK: return CUBLASLT_REDUCTION_SCHEME_MASK;
        case at::CuBLASReductionOption::DisallowReducedPrecisionAllowSplitK: return CUBLASLT_REDUCTION_SCHEME_COMPUTE_TYPE;
        default: return CUBLASLT_REDUCTION_SCHEME_NONE;
    }
}

// ta: A is stored [K,M]; tb: B is stored [N,K]; lda: elements between A's rows (0: none skipped)
void gemm(void* C, bool f32_out, const void* A, bool ta, const void* B, bool tb, const void* bias, int64_t M, int64_t N, int64_t K, const Tensor& on,
          int64_t lda = 0) {
    static thread_local std::map<GemmKey, std::unique_ptr<GemmPlan>> plans;
    constexpr size_t kMostPlans = 128;
    if (!on_16(A) || !on_16(B) || !on_16(C) || !on_16(bias) || lda % 8)                   // what the plans are chosen for
        throw std::runtime_error("dsqg: GEMM operands must start on 16 bytes");
    cublasLtHandle_t lt = at::cuda::getCurrentCUDABlasLtHandle();
    size_t space = at::cuda::getCUDABlasLtWorkspaceSize();
    const uint32_t schemes = reduction_schemes();
    const GemmKey key = {on.device().index(), M, N, K, (ta ? 1 : 0) | (tb ? 2 : 0) | (bias ? 4 : 0), f32_out, (int64_t)space, lda, schemes};
    if (plans.size() >= kMostPlans && !plans.count(key)) plans.clear();
    std::unique_ptr<GemmPlan>& slot = plans[key];
    if (!slot) {
        // cuBLAS is column-major: C^T[N,M] = op(B)^T . op(A)^T
        auto p = std::make_unique<GemmPlan>();
        lt_check(cublasLtMatmulDescCreate(&p->op, CUBLAS_COMPUTE_32F, CUDA_R_32F), "cublasLtMatmulDescCreate");
        const cublasOperation_t opb = tb ? CUBLAS_OP_T : CUBLAS_OP_N, opa = ta ? CUBLAS_OP_T : CUBLAS_OP_N;
        lt_check(cublasLtMatmulDescSetAttribute(p->op, CUBLASLT_MATMUL_DESC_TRANSA, &opb, sizeof opb), "cublasLtMatmulDescSetAttribute");
        lt_check(cublasLtMatmulDescSetAttribute(p->op, CUBLASLT_MATMUL_DESC_TRANSB, &opa, sizeof opa), "cublasLtMatmulDescSetAttribute");
        if (bias) {
            const cublasLtEpilogue_t e = CUBLASLT_EPILOGUE_BIAS;
            lt_check(cublasLtMatmulDescSetAttribute(p->op, CUBLASLT_MATMUL_DESC_EPILOGUE, &e, sizeof e), "cublasLtMatmulDescSetAttribute");
            lt_check(cublasLtMatmulDescSetAttribute(p->op, CUBLASLT_MATMUL_DESC_BIAS_POINTER, &bias, sizeof bias), "cublasLtMatmulDescSetAttribute");
        }
        lt_check(cublasLtMatrixLayoutCreate(&p->b, CUDA_R_16BF, tb ? K : N, tb ? N : K, tb ? K : N), "cublasLtMatrixLayoutCreate");
        lt_check(cublasLtMatrixLayoutCreate(&p->a, CUDA_R_16BF, ta ? M : K, ta ? K : M, lda ? lda : ta ? M : K), "cublasLtMatrixLayoutCreate");
        lt_check(cublasLtMatrixLayoutCreate(&p->c, f32_out ? CUDA_R_32F : CUDA_R_16BF, N, M, N), "cublasLtMatrixLayoutCreate");
        cublasLtMatmulPreference_t pref;
        lt_check(cublasLtMatmulPreferenceCreate(&pref), "cublasLtMatmulPreferenceCreate");
        const uint32_t align = 16;
        cublasLtMatmulPreferenceSetAttribute(pref, CUBLASLT_MATMUL_PREF_REDUCTION_SCHEME_MASK, &schemes, sizeof schemes);
        cublasLtMatmulPreferenceSetAttribute(pref, CUBLASLT_MATMUL_PREF_MAX_WORKSPACE_BYTES, &space, sizeof space);
        for (auto attr : {CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_A_BYTES, CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_B_BYTES, CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_C_BYTES,
                          CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_D_BYTES})
            cublasLtMatmulPreferenceSetAttribute(pref, attr, &align, sizeof align);
        cublasLtMatmulHeuristicResult_t best;
        int found = 0;
        const cublasStatus_t st = cublasLtMatmulAlgoGetHeuristic(lt, p->op, p->b, p->a, p->c, p->c, pref, 1, &best, &found);
        cublasLtMatmulPreferenceDestroy(pref);
        lt_check(st == CUBLAS_STATUS_SUCCESS && !found ? CUBLAS_STATUS_NOT_SUPPORTED : st, "cublasLtMatmulAlgoGetHeuristic");
        p->algo = best.algo; p->workspace = best.workspaceSize;
        slot = std::move(p);
    }
    GemmPlan& p = *slot;
    if (bias) lt_check(cublasLtMatmulDescSetAttribute(p.op, CUBLASLT_MATMUL_DESC_BIAS_POINTER, &bias, sizeof bias), "cublasLtMatmulDescSetAttribute");
    const float one = 1.f, zero = 0.f;
    lt_check(cublasLtMatmul(lt, p.op, &one, B, p.b, A, p.a, &zero, C, p.c, C, p.c, &p.algo, p.workspace ? at::cuda::getCUDABlasLtWorkspace() : nullptr,
                            p.workspace, static_cast<cudaStream_t>(stream_of(on))), "cublasLtMatmul");
}
// X[M,K] . W[N,K]^T + bias -> bf16 [M,N]
Tensor linear(const Tensor& X, const void* W, const void* bias, int64_t M, int64_t N, int64_t K) {
    Tensor C = new_tensor({M, N}, at::kBFloat16, X);
    gemm(ptr(C), false, ptr(X), false, W, true, bias, M, N, K, X);
    return C;
}
// dY[M,N] . W[N,K] -> [M,K]
Tensor grad_input(const Tensor& dY, const void* W, int64_t M, int64_t N, int64_t K, bool f32_out) {
    Tensor C = new_tensor({M, K}, f32_out ? at::kFloat : at::kBFloat16, dY);
    gemm(ptr(C), f32_out, ptr(dY), false, W, false, nullptr, M, K, N, dY);
    return C;
}
// dY[M,N]^T . X[M,K] -> fp32 [N,K]
Tensor grad_weight(const Tensor& dY, const Tensor& X, int64_t M, int64_t N, int64_t K) {
    Tensor C = new_tensor({N, K}, at::kFloat, dY);
    gemm(ptr(C), true, ptr(dY), true, ptr(X), false, nullptr, N, K, M, dY);
    return C;
}

// Weight and bias gradients of two projections over the same M rows in one launch (csrc/dsqg_wgrad.cu) instead of a GEMM each and their
// column sums.  Both sides of the line, us (M rows, two products [4 D, D] and [D, D]): D 256: M 1,024 7.6 against 9.8, 16,384 23.1 : 49.5,
// 65,536 70 : 107; D 128: 6.4 : 9.5, 18.4 : 39.9, 55.5 : 83.  Its error against 64 bits is at most the GEMMs', mostly a half to a sixth of it.  At D 512
// 16,384 rows it still wins (51 : 73), but not at 384 (125 : 121 with [2 D, D] and 65,536 rows), and above 512 it loses: more tiles than clusters that
// run at once.  The limit of 65,536 rows is one of precision: a block's chain of running sums grows with the rows.  Relative error against 64 bits, this
// kernel : GEMMs, D 256: 65,536 rows 1.2e-5 : 1.9e-5, 131,072 2.5e-5 : 1.8e-5, 262,144 5.0e-5 : 3.6e-5 (D 128 9.1e-6 : 1.7e-5, 1.9e-5 : 1.8e-5, 3.8e-5 : 3.1e-5; D 192
// 1.2e-5 : 1.2e-5, 2.5e-5 : 2.2e-5, 5.0e-5 : 3.2e-5), although it would be faster there too: 131,072 rows 132 us : 94 + 90 for the sums, 262,144 273 : 177 + 200.  The sums are split, so a caller who rules splits
// out (reduction_schemes) gets the GEMMs.
bool one_launch_weight_grads(int64_t M, int64_t D) {
    return D >= 128 && D <= 256 && D % 64 == 0 && M <= 65536 && reduction_schemes() != CUBLASLT_REDUCTION_SCHEME_NONE;
}
struct WeightGrad { const void* dy; int64_t ld; int64_t cols; const void* x; float* dw; float* sums; };
void weight_grads(const std::array<WeightGrad, 2>& jobs, int count, int64_t M, int64_t D, const Tensor& on) {
    const void *dy[2], *x[2]; long long ld[2]; int cols[2]; float *dw[2], *sums[2];
    for (int k = 0; k < count; ++k) {
        dy[k] = jobs[k].dy; x[k] = jobs[k].x; ld[k] = jobs[k].ld; cols[k] = (int)jobs[k].cols; dw[k] = jobs[k].dw; sums[k] = jobs[k].sums;
    }
    const int status = dsqg_weight_grads(dy, ld, cols, x, dw, sums, count, M, (int)D, stream_of(on));
    if (status != DSQG_ERR_UNSUPPORTED) return check(status, "dsqg_weight_grads");
    // a driver that makes no tensor maps: GEMMs and column sums into the same places
    const void* sp[2]; long long sld[2]; int sc[2]; float* to[2];
    int n = 0;
    for (int k = 0; k < count; ++k) {
        gemm(dw[k], true, dy[k], true, x[k], false, nullptr, cols[k], D, M, on, ld[k] == cols[k] ? 0 : ld[k]);
        if (sums[k]) { sp[n] = dy[k]; sld[n] = ld[k]; sc[n] = cols[k]; to[n] = sums[k]; ++n; }
    }
    if (n) check(dsqg_column_sums(sp, sld, sc, to, n, M, stream_of(on)), "dsqg_column_sums");
}

// fp32 tensors as bf16 back to back in one buffer, in one launch; at[k]: where the k-th begins (elements).
struct Bf16Pack {
    Tensor buf;
    std::vector<int64_t> at;
    const char* operator[](int k) const { return static_cast<const char*>(buf.data_ptr()) + 2 * at[k]; }
};
Bf16Pack cast_bf16(std::initializer_list<Tensor> src0) {
    Bf16Pack p;
    std::vector<Tensor> src;
    int64_t total = 0;
    for (const Tensor& t : src0) { src.push_back(aligned(f32c(t))); p.at.push_back(total); total += t.numel(); }
    p.buf = new_tensor({total}, at::kBFloat16, src[0]);
    const float* sp[DSQG_CAST_MAX]; void* dp[DSQG_CAST_MAX]; long long n[DSQG_CAST_MAX];
    for (size_t k = 0; k < src.size(); ++k) { sp[k] = fptr(src[k]); dp[k] = const_cast<char*>(p[(int)k]); n[k] = src[k].numel(); }
    check(dsqg_cast_bf16(sp, dp, n, (int)src.size(), stream_of(p.buf)), "dsqg_cast_bf16");
    return p;
}

// A vector or row-major matrix inside a flat buffer (a tensor on the same storage; a dispatched at::as_strided costs three times as much)
Tensor part(const Tensor& buf, at::IntArrayRef sizes, int64_t first) {
    Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(buf.storage()), buf.key_set(), buf.dtype());
    t.unsafeGetTensorImpl()->set_storage_offset(buf.storage_offset() + first);
    t.unsafeGetTensorImpl()->set_sizes_contiguous(sizes);
    return t;
}

struct Columns { const void* p; int64_t ld; int cols; };
// Column sums of bf16 matrices of `rows` rows, back to back; those without columns are left out.
Tensor column_sums(std::initializer_list<Columns> ms, int64_t rows, const Tensor& on) {
    int64_t total = 0;
    for (const Columns& m : ms) total += m.cols;
    if (!total) return Tensor();
    Tensor buf = new_tensor({total}, at::kFloat, on);
    const void* sp[DSQG_SUM_MAX]; long long ld[DSQG_SUM_MAX]; int cols[DSQG_SUM_MAX]; float* dp[DSQG_SUM_MAX];
    int k = 0;
    int64_t o = 0;
    for (const Columns& m : ms) {
        if (!m.cols) continue;
        sp[k] = m.p; ld[k] = m.ld; cols[k] = m.cols; dp[k] = fptr(buf) + o;
        o += m.cols; ++k;
    }
    check(dsqg_column_sums(sp, ld, cols, dp, k, rows, stream_of(on)), "dsqg_column_sums");
    return buf;
}

// [B,H,N,HD] view of columns [first, first + H*HD) of a row-major matrix of B*N rows, ld elements apart
Tensor heads_view(const Tensor& m, int64_t B, int64_t H, int64_t N, int64_t HD, int64_t ld, int64_t first) {
    return at::as_strided(m, {B, H, N, HD}, {N * ld, HD, ld, 1}, m.storage_offset() + first);
}
// The row stride of such a view (0: it is none).
int64_t heads_stride(const Tensor& t) {
    const int64_t H = t.size(1), N = t.size(2), HD = t.size(3), ld = t.stride(2);
    const bool ok = t.stride(3) == 1 && (H == 1 || t.stride(1) == HD) && ld >= H * HD && ld % 8 == 0 && (t.size(0) == 1 || t.stride(0) == N * ld) &&
                    on_16(t.data_ptr());
    return ok ? ld : 0;
}
Tensor rows_of(const Tensor& t) {        // [B,H,N,HD] -> [B*N, H*HD] bf16
    return aligned(t.permute({0, 2, 1, 3}).reshape({t.size(0) * t.size(2), t.size(1) * t.size(3)}).to(at::kBFloat16).contiguous());
}

// (k_delta, v_delta) of the interference block (train/train_2048_condU.py:277-295)
struct InterferenceNode : torch::autograd::Function<InterferenceNode> {
    static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& gamma, const Tensor& beta, const Tensor& wg, const Tensor& bg,
                                 const Tensor& wk, const Tensor& bk, const Tensor& wv, const Tensor& bv, double eps, int64_t H) {
        const NoAutocast no_autocast;
        const c10::cuda::CUDAGuard guard(x.device());
        const int64_t B = x.size(0), N = x.size(1), D = x.size(2), M = B * N;
        const Tensor xc = aligned(f32c(x)), gam = aligned(f32c(gamma));
        // the modules' own kernel, and so their bits: the deltas round as theirs do, and with them the gradients that nearly cancel
        const auto [xi, mean, rstd] = at::native_layer_norm(xc, {D}, gam, aligned(f32c(beta)), eps);
        const Bf16Pack w = cast_bf16({wg, wk, wv, bg, bk, bv, xi});               // wk, wv and bk, bv are one matrix and one vector
        const Tensor xib = part(w.buf, {M, D}, w.at[6]), g = linear(xib, w[0], w[3], M, D, D);
        Tensor pool = new_like(xi), inter = new_like(g);
        check(dsqg_gated_mean(fptr(xi), ptr(g), fptr(pool), ptr(inter), (int)B, (int)N, (int)D, stream_of(x)), "dsqg_gated_mean");
        const Tensor kv = linear(inter, w[1], w[4], M, 2 * D, D);
        ctx->save_for_backward({xc, gam, mean, rstd, xib, pool, g, inter, w.buf});
        ctx->saved_data["x_type"] = (int64_t)x.scalar_type();
        return {heads_view(kv, B, H, N, D / H, 2 * D, 0), heads_view(kv, B, H, N, D / H, 2 * D, D)};
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        return backward_body(grads[0].defined() ? grads[0] : grads[1], [&] { return run(ctx, grads); });
    }
    static variable_list run(AutogradContext* ctx, const variable_list& grads) {
        const NoAutocast no_autocast;
        const variable_list s = ctx->get_saved_variables();
        const Tensor &x = s[0], &gam = s[1], &mean = s[2], &rstd = s[3], &xib = s[4], &pool = s[5], &g = s[6], &inter = s[7], &w = s[8];
        const c10::cuda::CUDAGuard guard(x.device());
        const int64_t D = x.size(2), M = x.size(0) * x.size(1);
        // what is asked for, of x, gamma, beta, wg, bg, wk, bk, wv, bv
        const auto need = [&](size_t i) { return ctx->needs_input_grad(i); };
        const bool n_norm = need(0) || need(1) || need(2), n_in = n_norm || need(3) || need(4), n_wkv = need(5) || need(7), n_bkv = need(6) || need(8);
        // [M, 2 D]: the gradients of an attention layer lie like that already
        Tensor dkv;
        const void* dp = nullptr;
        int64_t ld = 0;
        const Tensor &dk = grads[0], &dv = grads[1];
        if (dk.defined() && dv.defined() && dk.scalar_type() == at::kBFloat16 && dv.scalar_type() == at::kBFloat16) {
            ld = heads_stride(dk);
            if (ld >= 2 * D && heads_stride(dv) == ld && static_cast<char*>(ptr(dv)) == static_cast<char*>(ptr(dk)) + 2 * D) dp = ptr(dk);
        }
        if (!dp) {
            const auto half = [&](const Tensor& d) { return d.defined() ? rows_of(d) : at::zeros({M, D}, xib.options()); };
            dkv = at::cat({half(dk), half(dv)}, 1);
            dp = ptr(dkv); ld = 2 * D;
        }
        void* stream = stream_of(x);
        const char* wb = static_cast<const char*>(ptr(w));
        Tensor dinter, dwkv, dg, dxi, dwg, dx, dgb;
        const bool one_launch = n_wkv && need(3) && one_launch_weight_grads(M, D);
        if (n_wkv) dwkv = new_tensor({2 * D, D}, at::kFloat, x);
        if (n_wkv && !one_launch) {
            gemm(ptr(dwkv), true, dp, true, ptr(inter), false, nullptr, 2 * D, D, M, x, ld);
        }
        if (n_in) {
            dinter = new_like(inter); dg = new_like(g); dxi = new_like(pool);
            gemm(ptr(dinter), false, dp, false, wb + 2 * D * D, false, nullptr, M, D, 2 * D, x, ld);
            check(dsqg_gated_mean_bwd(ptr(dinter), ptr(g), fptr(pool), ptr(dg), fptr(dxi), (int)x.size(0), (int)x.size(1), (int)D, stream), "dsqg_gated_mean_bwd");
        }
        const int64_t kv = need(4) ? D : 0;                    // where the sums of the two biases begin
        Tensor db;
        if (one_launch) {
            dwg = new_tensor({D, D}, at::kFloat, x);
            if (kv || n_bkv) db = new_tensor({kv + (n_bkv ? 2 * D : 0)}, at::kFloat, x);
            weight_grads({{{dp, ld, 2 * D, ptr(inter), fptr(dwkv), n_bkv ? fptr(db) + kv : nullptr}, {ptr(dg), D, D, ptr(xib), fptr(dwg), kv ? fptr(db) : nullptr}}},
                         2, M, D, x);
        } else {
            if (need(3)) dwg = grad_weight(dg, xib, M, D, D);
            db = column_sums({{ptr(dg), D, need(4) ? (int)D : 0}, {dp, ld, n_bkv ? (int)(2 * D) : 0}}, M, x);
        }
        if (n_norm) {
            const Tensor dxib = grad_input(dg, wb, M, D, D, false);
            dx = new_like(x); dgb = new_tensor({2 * D}, at::kFloat, x);
            const size_t bytes = dsqg_layer_norm_bwd_scratch_bytes(M, (int)D);
            const at::DataPtr scratch = scratch_for(bytes);
            check(dsqg_layer_norm_bwd_split(fptr(x), fptr(mean), fptr(rstd), fptr(gam), fptr(dxi), ptr(dxib), fptr(dx), fptr(dgb), scratch.get(), bytes, M, (int)D, stream),
                  "dsqg_layer_norm_bwd_split");
        }
        const auto piece = [&](bool wanted, const Tensor& buf, at::IntArrayRef sizes, int64_t first) { return wanted ? part(buf, sizes, first) : Tensor(); };
        return {need(0) ? like_param(dx, (at::ScalarType)ctx->saved_data["x_type"].toInt()) : Tensor(), piece(need(1), dgb, {D}, 0), piece(need(2), dgb, {D}, D),
                dwg, piece(need(4), db, {D}, 0), piece(need(5), dwkv, {D, D}, 0), piece(need(6), db, {D}, kv), piece(need(7), dwkv, {D, D}, D * D),
                piece(need(8), db, {D}, kv + D), Tensor(), Tensor()};
    }
};

// qkv projection -> (K/V injection) -> operator -> gate -> output projection (train/train_2048_condU.py:171-191).  The gate's
// projection is part of the qkv product (one GEMM over [q | k | v | gate] columns, one weight gradient, one input gradient).  Where the
// operator leaves copies of q, k, v for its backward, the forward's product is two GEMMs instead, so that only the gate's output is kept
// beside the copies (B32 N2048 dim 256: 100 MB less per layer than keeping all of it).
struct LayerNode : torch::autograd::Function<LayerNode> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, const std::optional<Tensor>& kd, const std::optional<Tensor>& vd, const Tensor& wqkv,
                          const Tensor& bqkv, const Tensor& wg, const Tensor& bg, const Tensor& wo, const Tensor& bo, const Tensor& pos_bias,
                          const std::optional<Tensor>& hg, const std::optional<Tensor>& se, const Offsets* off, int64_t H, bool with_grad) {
        const NoAutocast no_autocast;
        const c10::cuda::CUDAGuard guard(x.device());
        const int64_t B = x.size(0), N = x.size(1), D = x.size(2), M = B * N;
        const bool cast_x = x.scalar_type() == at::kFloat;
        const Bf16Pack w = cast_x ? cast_bf16({wqkv, wg, wo, bqkv, bg, bo, x}) : cast_bf16({wqkv, wg, wo, bqkv, bg, bo});
        const Tensor xb = cast_x ? part(w.buf, {M, D}, w.at[6]) : aligned(x.contiguous());
        const bool split = with_grad && dsqg_packed_keep_bytes((int)B, (int)H, (int)N, (int)(D / H));
        const int64_t cols = split ? 3 * D : 4 * D;
        const Tensor proj = linear(xb, w[0], w[3], M, cols, D);                   // bqkv and bg are one vector
        const Tensor gate = split ? linear(xb, w[1], w[4], M, D, D).view({B, N, D}) : Tensor();
        if (kd.has_value()) {
            Tensor k = *kd, v = *vd;
            int64_t ld = k.scalar_type() == at::kBFloat16 && v.scalar_type() == at::kBFloat16 ? heads_stride(k) : 0;
            if (!ld || heads_stride(v) != ld) { k = rows_of(k); v = rows_of(v); ld = D; }
            check(dsqg_inject_kv(ptr(proj), cols, ptr(k), ptr(v), ld, M, (int)D, stream_of(x)), "dsqg_inject_kv");
        }
        const PackedForward f = packed_forward(proj, B, N, H, D / H, cols, gate, pos_bias, opt(hg), opt(se), *off, with_grad);
        const Tensor out = linear(f.y, w[2], w[5], M, D, D).view({B, N, D});
        ctx->save_for_backward({xb, w.buf, f.keep.defined() ? Tensor() : proj, f.gate, f.pb, f.hg, f.se, f.y, f.lse, f.keep});
        ctx->saved_data["offsets"] = (int64_t)(intptr_t)off;
        ctx->saved_data["types"] = types_of(pos_bias, opt(hg), opt(se));
        ctx->saved_data["x_types"] = std::vector<int64_t>{(int64_t)x.scalar_type(), (int64_t)type_of(opt(kd)), (int64_t)type_of(opt(vd))};
        ctx->saved_data["inject"] = kd.has_value();
        return out;
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        return backward_body(grads[0], [&] { return run(ctx, grads[0]); });
    }
    static variable_list run(AutogradContext* ctx, const Tensor& dy0) {
        const NoAutocast no_autocast;
        const variable_list s = ctx->get_saved_variables();
        const Tensor &xb = s[0], &w = s[1];
        const PackedForward f = {s[2], s[3], s[4], s[5], s[6], s[7], s[8], s[9]};
        const int64_t B = f.lse.size(0), H = f.lse.size(1), N = f.lse.size(2), D = f.y.size(2), M = B * N, HD = D / H;
        const c10::cuda::CUDAGuard guard(xb.device());
        const Tensor dy = aligned(bf16c(dy0));
        const char* wb = static_cast<const char*>(ptr(w));
        // what is asked for; edges exist for the tensors that were given
        const auto xt = ctx->saved_data["x_types"].toIntVector();
        const bool inject = ctx->saved_data["inject"].toBool();
        size_t edge = 0;
        const auto need = [&](bool given = true) { return given && ctx->needs_input_grad(edge++); };
        const bool n_x = need(), n_k = need(inject), n_v = need(inject), n_wqkv = need(), n_bqkv = need(), n_wg = need(), n_bg = need(), n_wo = need(),
                   n_bo = need(), n_pb = need(), n_hg = need(f.hg.defined()), n_se = need(f.se.defined());
        Tensor dx, dk, dv, dw, dwo;
        PackedGrads g;
        // of the columns [qkv | gate], those from `first` on up to `last`
        const int64_t first = n_wqkv ? 0 : 3 * D, last = n_wg ? 4 * D : 3 * D, sum_first = n_bqkv ? 0 : 3 * D, sum_last = n_bg ? 4 * D : 3 * D;
        const int sums = (int)std::max<int64_t>(sum_last - sum_first, 0);
        const bool one_launch = last > first && n_wo && (!sums || (sum_first == first && sum_last == last)) && one_launch_weight_grads(M, D);
        if (n_wo && !one_launch) dwo = grad_weight(dy, f.y, M, D, D);
        if (n_x || n_k || n_v || n_wqkv || n_bqkv || n_wg || n_bg || n_pb || n_hg || n_se)
            g = packed_backward(f, grad_input(dy, wb + 2 * 4 * D * D, M, D, D, false), 4 * D, offsets_of(ctx));
        const auto column = [&](int64_t c) { return static_cast<const char*>(ptr(g.dproj)) + 2 * c; };
        if (last > first) dw = new_tensor({last - first, D}, at::kFloat, dy);
        if (last > first && !one_launch) {
            gemm(ptr(dw), true, column(first), true, ptr(xb), false, nullptr, last - first, D, M, dy, 4 * D);
        }
        Tensor db;
        if (one_launch) {
            dwo = new_tensor({D, D}, at::kFloat, dy);
            if (sums || n_bo) db = new_tensor({sums + (n_bo ? D : 0)}, at::kFloat, dy);
            weight_grads({{{column(first), 4 * D, last - first, ptr(xb), fptr(dw), sums ? fptr(db) : nullptr},
                           {ptr(dy), D, D, ptr(f.y), fptr(dwo), n_bo ? fptr(db) + sums : nullptr}}}, 2, M, D, dy);
        } else db = column_sums({{sums ? column(sum_first) : nullptr, 4 * D, sums}, {ptr(dy), D, n_bo ? (int)D : 0}}, M, xb);
        if (n_x) {
            const auto t = (at::ScalarType)xt[0];
            dx = like_param(grad_input(g.dproj, wb, M, 4 * D, D, t == at::kFloat).view({B, N, D}), t);
        }
        if (n_k) dk = like_param(heads_view(g.dproj, B, H, N, HD, 4 * D, D), (at::ScalarType)xt[1]);
        if (n_v) dv = like_param(heads_view(g.dproj, B, H, N, HD, 4 * D, 2 * D), (at::ScalarType)xt[2]);
        const auto piece = [&](bool wanted, const Tensor& buf, at::IntArrayRef sizes, int64_t at) { return wanted ? part(buf, sizes, at) : Tensor(); };
        return {dx, dk, dv, piece(n_wqkv, dw, {3 * D, D}, 0), piece(n_bqkv, db, {3 * D}, 0), piece(n_wg, dw, {D, D}, (3 * D - first) * D), piece(n_bg, db, {D}, 3 * D - sum_first),
                dwo, piece(n_bo, db, {D}, sums), n_pb ? like_param(g.dpb, type_at(ctx, 0)) : Tensor(), n_hg ? like_param(g.dhg, type_at(ctx, 1)) : Tensor(),
                n_se ? like_param(g.dse, type_at(ctx, 2)) : Tensor(), Tensor(), Tensor(), Tensor()};
    }
};

// The nodes serve fp32 parameters under bf16 autocast.
bool layer_applies(const Tensor& x, const std::vector<Tensor>& params) {
    if (!x.is_cuda() || x.dim() != 3 || x.size(0) < 1 || x.size(1) < 1 || (x.scalar_type() != at::kFloat && x.scalar_type() != at::kBFloat16)) return false;
    if (!at::autocast::is_autocast_enabled(at::kCUDA) || at::autocast::get_autocast_dtype(at::kCUDA) != at::kBFloat16) return false;
    for (const Tensor& p : params)
        if (p.scalar_type() != at::kFloat || p.device() != x.device()) return false;
    return true;
}

std::tuple<Tensor, Tensor> interference(const Tensor& x, const Tensor& gamma, const Tensor& beta, const Tensor& wg, const Tensor& bg, const Tensor& wk,
                                        const Tensor& bk, const Tensor& wv, const Tensor& bv, double eps, int64_t H) {
    py::gil_scoped_release no_gil;
    const variable_list r = InterferenceNode::apply(x, gamma, beta, wg, bg, wk, bk, wv, bv, eps, H);
    return {r[0], r[1]};
}
Tensor layer(const Tensor& x, const std::optional<Tensor>& kd, const std::optional<Tensor>& vd, const Tensor& wqkv, const Tensor& bqkv, const Tensor& wg,
             const Tensor& bg, const Tensor& wo, const Tensor& bo, const Tensor& pb, const std::optional<Tensor>& hg, const std::optional<Tensor>& se,
             const Offsets* off, int64_t H) {
    py::gil_scoped_release no_gil;
    return LayerNode::apply(x, kd, vd, wqkv, bqkv, wg, bg, wo, bo, pb, hg, se, off, H, at::GradMode::is_enabled());
}

// ------------------------------------------------------------------------------------ decode
struct StepParams { Tensor pb, hg, se; };

void check_step(const char* who, const Tensor& q, const Tensor& k, const Tensor& v, at::ScalarType dt, int64_t S, int64_t H, int64_t D,
                const Tensor& ring, const Tensor& head, const Tensor& fill, const Tensor& pb, const Tensor& hg, const Tensor& se, int J) {
    check_device(who, q, {&k, &v, &ring, &head, &fill, &pb, &hg, &se});
    const char* names[3] = {"q", "k_new", "v_new"};
    const Tensor* ts[3] = {&q, &k, &v};
    for (int i = 0; i < 3; ++i)
        if (!shape_is(*ts[i], {S, H, D}) || ts[i]->scalar_type() != dt || !ts[i]->is_contiguous())
            throw py::value_error(std::string(who) + ": " + names[i] + " must be contiguous [" + std::to_string(S) + "," + std::to_string(H) + "," +
                                  std::to_string(D) + "] " + toString(dt));
    if (head.scalar_type() != at::kInt || !shape_is(head, {S})) throw py::value_error(std::string(who) + ": head must be int32 [S]");
    if (fill.defined() && (fill.scalar_type() != at::kInt || !shape_is(fill, {S}))) throw py::value_error(std::string(who) + ": fill must be int32 [S]");
    if (!shape_is(pb, {J, H})) throw py::value_error(std::string(who) + ": pos_bias must be [" + std::to_string(J) + "," + std::to_string(H) + "]");
}

Tensor decode_step(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& k_ring, const Tensor& v_ring, const Tensor& head,
                   const Tensor& pos_bias, const std::optional<Tensor>& hg, const std::optional<Tensor>& se, const Offsets* off,
                   const std::optional<Tensor>& fill0, const std::optional<Tensor>& out0, bool overlap) {
    if (k_ring.dim() != 4) throw py::value_error("dsqg_decode: k_ring and v_ring must be contiguous [S,H,R,D]");
    const int64_t S = k_ring.size(0), H = k_ring.size(1), R = k_ring.size(2), D = k_ring.size(3);
    const Tensor fill = opt(fill0);
    check_step("dsqg_decode", q, k, v, k_ring.scalar_type(), S, H, D, k_ring, head, fill, pos_bias, opt(hg), opt(se), off->J());
    check_device("dsqg_decode", q, {&v_ring});
    if (v_ring.sizes() != k_ring.sizes() || !k_ring.is_contiguous() || !v_ring.is_contiguous())
        throw py::value_error("dsqg_decode: k_ring and v_ring must be contiguous [S,H,R,D]");
    const StepParams p = {f32c(pos_bias), f32c(opt(hg)), f32c(opt(se))};
    const c10::cuda::CUDAGuard guard(q.device());
    Tensor out = out0.has_value() ? *out0 : new_like(q);
    check((overlap ? dsqg_decode_overlapped : dsqg_decode)(
              ptr(q), ptr(k), ptr(v), ptr(k_ring), ptr(v_ring), static_cast<const int32_t*>(ptr(head)), static_cast<const int32_t*>(ptr(fill)),
              fptr(p.pb), fptr(p.se), fptr(p.hg), off->v.data(), off->J(), (int)R, ptr(out), (int)S, (int)H, (int)D, dtype_code(q), stream_of(q)),
          "dsqg_decode");
    return out;
}

// kv_ring [S,H,R,2,D], or the rings of all layers [L,S,H,R,2,D] and the layer to use
Tensor decode_step_kv(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& kv, std::optional<int64_t> layer0, const Tensor& head, const Tensor& pos_bias,
                      const std::optional<Tensor>& hg, const std::optional<Tensor>& se, const Offsets* off,
                      const std::optional<Tensor>& fill0, const std::optional<Tensor>& out0, bool overlap) {
    const int64_t lead = layer0.has_value() ? 1 : 0;
    if (kv.dim() != 5 + lead || kv.size(3 + lead) != 2 || !kv.is_contiguous()) throw py::value_error("dsqg_decode_kv: kv_ring must be contiguous [S,H,R,2,D]");
    const int64_t layer = !lead ? 0 : *layer0 < 0 ? *layer0 + kv.size(0) : *layer0;
    if (lead && (layer < 0 || layer >= kv.size(0))) throw py::index_error("dsqg_decode_kv: no such layer");
    const int64_t S = kv.size(lead), H = kv.size(1 + lead), R = kv.size(2 + lead), D = kv.size(4 + lead);
    const Tensor fill = opt(fill0);
    check_step("dsqg_decode_kv", q, k, v, kv.scalar_type(), S, H, D, kv, head, fill, pos_bias, opt(hg), opt(se), off->J());
    const StepParams p = {f32c(pos_bias), f32c(opt(hg)), f32c(opt(se))};
    const c10::cuda::CUDAGuard guard(q.device());
    Tensor out = out0.has_value() ? *out0 : new_like(q);
    char* ring = static_cast<char*>(kv.data_ptr()) + (lead ? layer * kv.stride(0) * kv.element_size() : 0);
    check(dsqg_decode_kv(ptr(q), ptr(k), ptr(v), ring, static_cast<const int32_t*>(ptr(head)), static_cast<const int32_t*>(ptr(fill)),
                         fptr(p.pb), fptr(p.se), fptr(p.hg), off->v.data(), off->J(), (int)R, ptr(out), (int)S, (int)H, (int)D, dtype_code(q),
                         stream_of(q), overlap), "dsqg_decode_kv");
    return out;
}

// (head + 1) mod R and min(fill + 1, R) as new tensors
std::tuple<Tensor, Tensor> ring_advance(const Tensor& head0, const Tensor& fill0, int64_t R) {
    const Tensor head = head0.to(at::kInt).contiguous(), fill = fill0.to(at::kInt).contiguous();
    const c10::cuda::CUDAGuard guard(head.device());
    Tensor h = new_like(head), f = new_like(fill);
    check(dsqg_ring_advance(static_cast<const int32_t*>(ptr(head)), static_cast<const int32_t*>(ptr(fill)), static_cast<int32_t*>(ptr(h)),
                            static_cast<int32_t*>(ptr(f)), (int)head.numel(), (int)R, stream_of(head)), "dsqg_ring_advance");
    return {h, f};
}

}  // namespace

PYBIND11_MODULE(_dsqg_torch, m) {
    py::class_<Offsets, std::unique_ptr<Offsets, py::nodelete>>(m, "Offsets").def_property_readonly("J", &Offsets::J);
    m.def("offsets", &intern_offsets, py::return_value_policy::reference);
    m.def("padded_head_dim", [](int64_t D, bool bf16, const Offsets* off, bool has_se) { return padded_head_dim(D, bf16, *off, has_se); });
    m.def("attention", &attention);
    m.def("forward_lse", &forward_lse);
    m.def("attention_packed", &attention_packed);
    m.def("layer_applies", &layer_applies);
    m.def("reduction_schemes", &reduction_schemes);
    m.def("interference", &interference);
    m.def("layer", &layer);
    m.def("causal_mean", &causal_mean);
    m.def("decode_step", &decode_step);
    m.def("decode_step_kv", &decode_step_kv);
    m.def("ring_advance", &ring_advance);
}
