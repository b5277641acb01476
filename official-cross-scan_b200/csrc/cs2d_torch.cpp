// Native host path of the PyTorch operators: argument checks, allocation, launch and the autograd nodes.
//
// A call of the operator on a small map costs a few tens of microseconds on the GPU; the checks, the
// problem description and the allocations cost several times that when they run in Python (measured on the
// 8x8 fp32 training step: 231 us per pass through ctypes and a Python autograd function, the two kernels
// about 20 us of it).  They live here instead, above the same C ABI (include/cs2d.h); cs2d/ops.py and
// cs2d/cross.py keep the public functions and their documentation.  The checks follow the reference host
// binding (src/cusoflex/selective_scan_oflex.cpp:179-440).
//
// Buffers of one backward: the parameter gradients (dA | dD | ddelta_bias | dA_decay) are one zero-filled
// fp32 buffer; the fp32 sums behind 16-bit dB and dC are another one (one fill instead of two).  Small
// problems take one allocation and one fill for all of these and the scratch (see BwdBuffers).  The backward
// runs on a thread of the autograd engine that has just been woken: every call of the tensor library costs
// twice there what it costs in a warm loop (measured 45 us for what takes 22 us on the calling thread).
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/extension.h>

#include <tuple>
#include <vector>

#include "../../include/cs2d.h"

namespace {

using at::Tensor;
using OptT = std::optional<Tensor>;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

#define CS2D_CHECK(cond, ...)                                  \
    do {                                                       \
        if (C10_UNLIKELY(!(cond))) fail_with(c10::str(__VA_ARGS__)); \
    } while (0)

[[noreturn]] void fail_with(const std::string &msg) { throw std::runtime_error(msg); }

int dtype_code(at::ScalarType t) {
    switch (t) {
        case at::kFloat: return CS2D_F32;
        case at::kHalf: return CS2D_F16;
        case at::kBFloat16: return CS2D_BF16;
        default: return -1;
    }
}
bool inner_ok(const Tensor &t) { return t.stride(-1) == 1 || t.size(-1) == 1; }
bool given(const Tensor &t) { return t.defined(); }
Tensor opt(const OptT &t) { return t.has_value() ? *t : Tensor(); }
bool deterministic_mode() { return at::globalContext().deterministicAlgorithms(); }

struct Args {
    Tensor u, delta, A, B, C, D, bias, decay;
    bool softplus;
};

// Checks the tensors and fills the C ABI's problem.  shared_u: u holds the channels of ONE group, read by
// all groups (the four-corner operator).
cs2d_problem make_problem(const Args &a, at::ScalarType out_type, const char *who, bool shared_u) {
    const int code = dtype_code(a.u.scalar_type());
    CS2D_CHECK(code >= 0, who, " not implemented for input type '", a.u.scalar_type(), "'");
    CS2D_CHECK(a.A.scalar_type() == at::kFloat, "A must be float32");
    const auto ty = a.u.scalar_type();
    CS2D_CHECK(a.delta.scalar_type() == ty && a.B.scalar_type() == ty && a.C.scalar_type() == ty,
               "delta, B, C must have the dtype of u");
    const std::pair<const char *, const Tensor *> must[] = {{"u", &a.u}, {"delta", &a.delta}, {"A", &a.A}, {"B", &a.B}, {"C", &a.C}};
    for (const auto &m : must) CS2D_CHECK(m.second->is_cuda(), m.first, " must be a CUDA tensor");
    CS2D_CHECK(a.u.dim() == 4, "u must have shape (batch_size, dim, nrows, ncols)");
    CS2D_CHECK(inner_ok(a.u) && inner_ok(a.delta), "u and delta must be contiguous in the last dimension");
    const int64_t batch = a.u.size(0), nrows = a.u.size(2), ncols = a.u.size(3);
    int64_t dim = a.u.size(1);
    if (shared_u) {
        CS2D_CHECK(a.B.dim() == 5 && a.A.dim() == 2 && dim * a.B.size(1) == a.A.size(0), "u must have dim / n_groups channels");
        dim = a.A.size(0);
    }
    CS2D_CHECK(a.A.dim() == 2 && a.B.dim() == 5 && a.delta.dim() == 4, "A, B, delta have the wrong rank");
    const int64_t n = a.A.size(1), groups = a.B.size(1), ddim = a.delta.size(1);
    CS2D_CHECK(groups > 0 && dim % groups == 0, "dims should be dividable by n_groups");
    CS2D_CHECK(ddim > 0 && dim % ddim == 0, "dims should be dividable by delta_dim");
    CS2D_CHECK(n <= CS2D_MAX_DSTATE, "selective_scan only supports state dimension <= ", CS2D_MAX_DSTATE);
    CS2D_CHECK(a.delta.sizes() == at::IntArrayRef({batch, ddim, nrows, ncols}),
               "delta must have shape (batch_size, delta_dim, nrows, ncols)");
    CS2D_CHECK(a.A.size(0) == dim, "A must have shape (dim, dstate)");
    if (given(a.decay)) {
        CS2D_CHECK(a.decay.dim() == 1 && a.decay.size(0) == 1, "A_decay must have shape (1)");
        CS2D_CHECK(a.decay.scalar_type() == at::kFloat && a.decay.is_cuda(), "A_decay must be a float32 CUDA tensor");
    }
    CS2D_CHECK(a.B.sizes() == at::IntArrayRef({batch, groups, n, nrows, ncols}),
               "B must have shape (batch_size, n_groups, dstate, nrows, ncols)");
    CS2D_CHECK(inner_ok(a.B), "B must be contiguous in the last dimension");
    CS2D_CHECK(a.C.sizes() == at::IntArrayRef({batch, groups, n, nrows, ncols}),
               "C must have shape (batch_size, n_groups, dstate, nrows, ncols)");
    CS2D_CHECK(inner_ok(a.C), "C must be contiguous in the last dimension");
    if (given(a.D)) {
        CS2D_CHECK(a.D.scalar_type() == at::kFloat && a.D.is_cuda() && a.D.dim() >= 1 && inner_ok(a.D),
                   "D must be a contiguous float32 CUDA tensor");
        CS2D_CHECK(a.D.dim() == 1 && a.D.size(0) == dim, "D must have shape (dim)");
    }
    if (given(a.bias)) {
        CS2D_CHECK(a.bias.scalar_type() == at::kFloat && a.bias.is_cuda() && a.bias.dim() >= 1 && inner_ok(a.bias),
                   "delta_bias must be a contiguous float32 CUDA tensor");
        CS2D_CHECK(a.bias.dim() == 1 && a.bias.size(0) == ddim, "delta_bias must have shape (delta_dim)");
    }
    cs2d_problem p{};
    p.batch = (int32_t)batch; p.dim = (int32_t)dim; p.nrows = (int32_t)nrows; p.ncols = (int32_t)ncols;
    p.dstate = (int32_t)n; p.n_groups = (int32_t)groups; p.delta_dim = (int32_t)ddim;
    p.io_dtype = code; p.out_dtype = dtype_code(out_type); p.delta_softplus = a.softplus;
    p.u = a.u.const_data_ptr(); p.u_bs = a.u.stride(0); p.u_ds = a.u.stride(1); p.u_hs = a.u.stride(2);
    p.delta = a.delta.const_data_ptr();
    p.delta_bs = a.delta.stride(0); p.delta_ds = a.delta.stride(1); p.delta_hs = a.delta.stride(2);
    p.A = a.A.const_data_ptr<float>(); p.A_ds = a.A.stride(0); p.A_ns = a.A.stride(1);
    p.B = a.B.const_data_ptr(); p.B_bs = a.B.stride(0); p.B_gs = a.B.stride(1); p.B_ns = a.B.stride(2); p.B_hs = a.B.stride(3);
    p.C = a.C.const_data_ptr(); p.C_bs = a.C.stride(0); p.C_gs = a.C.stride(1); p.C_ns = a.C.stride(2); p.C_hs = a.C.stride(3);
    p.D = given(a.D) ? a.D.const_data_ptr<float>() : nullptr;
    p.delta_bias = given(a.bias) ? a.bias.const_data_ptr<float>() : nullptr;
    p.A_decay = given(a.decay) ? a.decay.const_data_ptr<float>() : nullptr;
    return p;
}

void raise_on(int rc, const char *what) {
    if (C10_UNLIKELY(rc != 0)) fail_with(c10::str("cs2d ", what, " failed (", rc, "): ", cs2d_last_error()));
}
Tensor f32(const Tensor &like, int64_t n) { return at::empty({n}, like.options().dtype(at::kFloat)); }
cudaStream_t stream_of(const Tensor &t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
void zero(const Tensor &t, int64_t n) {   // the first n floats, with one asynchronous memset
    if (n <= 0) return;
    const cudaError_t e = cudaMemsetAsync(t.data_ptr(), 0, (size_t)n * 4, stream_of(t));
    CS2D_CHECK(e == cudaSuccess, "cs2d: zero fill failed: ", cudaGetErrorString(e));
}
Tensor zeros_f32(const Tensor &like, int64_t n) {
    Tensor t = f32(like, n);
    zero(t, n);
    return t;
}
float *fp(const Tensor &t) { return given(t) ? t.data_ptr<float>() : nullptr; }

// ---- forward ---------------------------------------------------------------------------------------
// deterministic: a deterministic backward will read the state, which is then the one that it takes without a second forward
std::pair<Tensor, Tensor> scan_forward(const Args &a, bool out_float, bool keep_state, bool deterministic) {
    const auto ot = out_float ? at::kFloat : a.u.scalar_type();
    const cs2d_problem p = make_problem(a, ot, "selective_scan_fwd", false);
    cs2d_dirs o{};
    if (deterministic && keep_state && cs2d_bwd_det_scratch_bytes_dir(&p, nullptr) != 0) o.flags = CS2D_DIRS_TILE_STATE;
    const size_t nbytes = keep_state ? cs2d_saved_bytes_dir(&p, &o) : cs2d_fwd_only_scratch_bytes_dir(&p, nullptr);
    CS2D_CHECK(nbytes != 0, "cs2d forward: ", cs2d_last_error());
    const c10::cuda::CUDAGuard guard(a.u.device());
    Tensor out = at::empty(a.u.sizes(), a.u.options().dtype(ot)), state = f32(a.u, (int64_t)(nbytes / 4));
    const int rc = keep_state ? cs2d_fwd_dir(&p, &o, out.data_ptr(), out.stride(0), out.stride(1), out.stride(2), state.data_ptr(), stream_of(a.u))
                              : cs2d_fwd_only(&p, nullptr, out.data_ptr(), out.stride(0), out.stride(1), out.stride(2),
                                              state.data_ptr(), stream_of(a.u));
    raise_on(rc, "forward");
    return {out, state};
}

// Offsets of dA | dD | ddelta_bias | dA_decay in one flat fp32 buffer (ops.param_grad_layout); -1: absent
struct ParamLayout { int64_t dD, dbias, ddecay, total; };
ParamLayout param_layout(int64_t dim, int64_t n, bool has_D, bool has_bias, bool has_decay) {
    ParamLayout l{-1, -1, -1, dim * n};
    if (has_D) { l.dD = l.total; l.total += dim; }
    if (has_bias) { l.dbias = l.total; l.total += dim; }
    if (has_decay) { l.ddecay = l.total; l.total += 1; }
    return l;
}

struct Grads { Tensor du, ddelta, dA, dB, dC, dD, dbias, ddecay, dw; };

// A contiguous tensor on part of another one's storage (no view in autograd's eyes, a fifth of the cost of narrow + view)
Tensor part_of(const Tensor &t, int64_t offset, at::IntArrayRef sizes) {
    c10::Storage st = t.storage();
    Tensor r = at::detail::make_tensor<c10::TensorImpl>(std::move(st), t.key_set(), t.dtype());
    r.unsafeGetTensorImpl()->set_sizes_contiguous(sizes);
    r.unsafeGetTensorImpl()->set_storage_offset(t.storage_offset() + offset);
    return r;
}

// Device buffers of a backward: `nparam` floats of parameter gradients and the fp32 sums of dB and dC, zero-filled, and
// the scratch.  Up to 256 KB in all they are one allocation with one fill, and 16-bit dB and dC are rounded together:
// what a caller keeps then keeps no more than that alive.  Larger ones are buffers of their own: two tensors dB and dC
// that share no storage.
struct BwdBuffers {
    Tensor params, b, c, scratch;
    int64_t half = 0, off = -1;   // off: where dB starts in a shared buffer; dC follows `half` elements later
    float *dB, *dC;
    void *scratch_ptr;
    BwdBuffers(const Tensor &B, int64_t nparam, size_t scratch_bytes, bool share) {
        const int64_t n = B.numel(), head = (nparam + 7) & ~int64_t(7), ns = (int64_t)(scratch_bytes / 4);
        half = (n + 7) & ~int64_t(7);
        if (share && head + 2 * half + ns <= (1 << 16)) {
            off = head;
            params = f32(B, head + 2 * half + ns);
            zero(params, head + 2 * half);
            float *p = params.data_ptr<float>();
            dB = p + off; dC = dB + half; scratch_ptr = dC + half;
            return;
        }
        if (nparam > 0) params = zeros_f32(B, nparam);
        if (B.scalar_type() == at::kFloat) {
            b = zeros_f32(B, n); c = zeros_f32(B, n);
        } else {
            const Tensor flat = zeros_f32(B, 2 * half);
            b = part_of(flat, 0, {n}); c = part_of(flat, half, {n});
        }
        dB = b.data_ptr<float>(); dC = c.data_ptr<float>();
        scratch = f32(B, ns);
        scratch_ptr = scratch.data_ptr();
    }
    void result(const Tensor &B, Tensor &gB, Tensor &gC) {
        const auto ty = B.scalar_type();
        if (off >= 0) {
            const bool cast = ty != at::kFloat;
            const Tensor t = cast ? part_of(params, off, {2 * half}).to(ty) : params;
            gB = part_of(t, cast ? 0 : off, B.sizes());
            gC = part_of(t, (cast ? 0 : off) + half, B.sizes());
        } else {
            gB = (ty == at::kFloat ? b : b.to(ty)).view(B.sizes());
            gC = (ty == at::kFloat ? c : c.to(ty)).view(B.sizes());
        }
    }
};

void param_views(Grads &g, const Tensor &flat, const ParamLayout &l, int64_t dim, int64_t n) {
    g.dA = part_of(flat, 0, {dim, n});
    if (l.dD >= 0) g.dD = part_of(flat, l.dD, {dim});
    if (l.dbias >= 0) g.dbias = part_of(flat, l.dbias, {dim});
    if (l.ddecay >= 0) g.ddecay = part_of(flat, l.ddecay, {1});
}

Grads scan_backward(const Args &a, const Tensor &dout, const Tensor &state, const OptT &param_grads, bool deterministic) {
    CS2D_CHECK(dout.is_cuda(), "dout must be a CUDA tensor");
    CS2D_CHECK(dout.scalar_type() == a.u.scalar_type() || dout.scalar_type() == at::kFloat, "dout must have the input dtype or float32");
    CS2D_CHECK(dout.sizes() == a.u.sizes(), "dout must have shape (batch_size, dim, nrows, ncols)");
    CS2D_CHECK(inner_ok(dout), "dout must be contiguous in the last dimension");
    const cs2d_problem p = make_problem(a, dout.scalar_type(), "selective_scan_bwd", false);
    CS2D_CHECK(given(state), "the saved state x_v returned by fwd is required");
    cs2d_dirs o{};
    const size_t nbytes = cs2d_saved_bytes_dir(&p, &o);
    CS2D_CHECK(nbytes != 0, "cs2d backward: ", cs2d_last_error());
    if (state.numel() * 4 != (int64_t)nbytes) o.flags = CS2D_DIRS_TILE_STATE;   // written for a deterministic backward
    CS2D_CHECK(state.is_cuda() && state.scalar_type() == at::kFloat && state.is_contiguous() &&
               state.numel() * 4 == (int64_t)(o.flags ? cs2d_saved_bytes_dir(&p, &o) : nbytes),
               "x_v is not the saved state fwd returned for these inputs");
    const int64_t dim = p.dim, n = p.dstate;
    const ParamLayout l = param_layout(dim, n, given(a.D), given(a.bias), given(a.decay));
    const c10::cuda::CUDAGuard guard(a.u.device());
    const cudaStream_t st = stream_of(a.u);
    Grads g;
    g.du = at::empty(a.u.sizes(), a.u.options());
    g.ddelta = at::empty(a.u.sizes(), a.u.options());
    const bool own = !param_grads.has_value();   // (a caller that brings its own buffer - the dispatcher operators - wants no shared storage)
    BwdBuffers buf(a.B, own ? l.total : 0, deterministic ? cs2d_bwd_scratch_bytes(&p) : cs2d_bwd_scratch_bytes_dir(&p, &o), own);
    Tensor flat = buf.params;
    if (!own) {
        flat = *param_grads;
        CS2D_CHECK(flat.is_cuda() && flat.scalar_type() == at::kFloat && flat.is_contiguous() && flat.numel() == l.total,
                   "param_grads must be a flat float32 CUDA tensor of the layout size");
    }
    param_views(g, flat, l, dim, n);
    if (deterministic) {
        const size_t ndet = cs2d_bwd_det_scratch_bytes_dir(&p, &o);
        CS2D_CHECK(ndet != 0, "cs2d backward has no deterministic implementation for this shape: ", cs2d_last_error());
        const Tensor det = f32(a.u, (int64_t)(ndet / 4));
        raise_on(cs2d_bwd_det(&p, &o, dout.const_data_ptr(), dout.stride(0), dout.stride(1), dout.stride(2), state.const_data_ptr(),
                              buf.scratch_ptr, det.data_ptr(), g.du.data_ptr(), g.ddelta.data_ptr(), fp(g.dA), buf.dB, buf.dC,
                              fp(g.dD), fp(g.dbias), fp(g.ddecay), st), "backward");
    } else {
        raise_on(cs2d_bwd_dir(&p, &o, dout.const_data_ptr(), dout.stride(0), dout.stride(1), dout.stride(2), state.const_data_ptr(),
                          buf.scratch_ptr, g.du.data_ptr(), g.ddelta.data_ptr(), fp(g.dA), buf.dB, buf.dC, fp(g.dD), fp(g.dbias),
                          fp(g.ddecay), st), "backward");
    }
    if (p.delta_dim != dim) {
        const int64_t rep = dim / p.delta_dim;
        g.ddelta = g.ddelta.view({a.u.size(0), p.delta_dim, rep, a.u.size(2), a.u.size(3)}).sum(2);
        if (given(g.dbias)) g.dbias = g.dbias.view({p.delta_dim, rep}).sum(1);
    }
    buf.result(a.B, g.dB, g.dC);
    return g;
}

// ---- four-corner operator --------------------------------------------------------------------------
void cross_check(const Args &a, const Tensor &w) {
    CS2D_CHECK(a.u.dim() == 4 && a.B.dim() == 5 && a.A.dim() == 2 && a.delta.dim() == 4 && w.dim() == 2,
               "expected delta (b, K*D, h, w), A (K*D, n), w (K, D)");
    const int64_t d = a.u.size(1), K = a.B.size(1);
    CS2D_CHECK(a.delta.size(1) == K * d && a.A.size(0) == K * d && w.size(0) == K && w.size(1) == d,
               "expected delta (b, K*D, h, w), A (K*D, n), w (K, D)");
}
cs2d_dirs make_dirs(int64_t K, int shared, bool serial, const Tensor &w, float *dw) {
    cs2d_dirs o{};
    for (int64_t k = 0; k < K && k < 32; ++k) {   // direction k: bit 1 of k mirrors the rows, bit 0 the columns
        if (k & 2) o.flip_rows_mask |= 1u << k;
        if (k & 1) o.flip_cols_mask |= 1u << k;
    }
    o.shared_input = shared; o.flags = serial ? CS2D_DIRS_SERIAL : 0;
    o.merge_w = w.const_data_ptr<float>(); o.merge_dw = dw;
    return o;
}
// reproducible form, rows of at most 256 columns: the kernel writes the merged image; otherwise it adds onto it
Tensor merged_image(const Tensor &u, bool serial) {
    if (serial && u.size(3) <= 256) return at::empty(u.sizes(), u.options().dtype(at::kFloat));
    return zeros_f32(u, u.numel()).view(u.sizes());
}
std::pair<Tensor, Tensor> cross_forward(const Args &a, const Tensor &w, bool serial, bool keep_state) {
    const cs2d_problem p = make_problem(a, at::kFloat, "cross_scan_fwd", true);
    const Tensor wf = w.to(at::kFloat).contiguous();
    const cs2d_dirs o = make_dirs(p.n_groups, 1, serial, wf, nullptr);
    const size_t nbytes = keep_state ? cs2d_saved_bytes_dir(&p, &o) : cs2d_fwd_only_scratch_bytes_dir(&p, &o);
    CS2D_CHECK(nbytes != 0, "cs2d forward: ", cs2d_last_error());
    const c10::cuda::CUDAGuard guard(a.u.device());
    Tensor out = merged_image(a.u, serial), state = f32(a.u, (int64_t)(nbytes / 4));
    raise_on((keep_state ? cs2d_fwd_dir : cs2d_fwd_only)(&p, &o, out.data_ptr(), out.stride(0), out.stride(1), out.stride(2),
                                                         state.data_ptr(), stream_of(a.u)), "forward");
    return {out, state};
}
Grads cross_backward(const Args &a, const Tensor &w, const Tensor &dy, const Tensor &state, bool serial) {
    const cs2d_problem p = make_problem(a, dy.scalar_type(), "cross_scan_bwd", true);
    CS2D_CHECK(p.out_dtype >= 0 && dy.is_cuda() && inner_ok(dy) && dy.sizes() == a.u.sizes(), "dy must be the gradient of the merged image");
    const int64_t dim = p.dim, n = p.dstate;
    const Tensor wf = w.to(at::kFloat).contiguous();
    const ParamLayout l = param_layout(dim, n, given(a.D), given(a.bias), given(a.decay));
    const c10::cuda::CUDAGuard guard(a.u.device());
    Grads g;
    cs2d_dirs o = make_dirs(p.n_groups, 3, serial, wf, nullptr);   // u and dy are shared by the directions
    CS2D_CHECK(state.is_cuda() && state.scalar_type() == at::kFloat && state.is_contiguous() &&
               state.numel() * 4 == (int64_t)cs2d_saved_bytes_dir(&p, &o), "the saved state is not the one the forward returned for these inputs");
    BwdBuffers buf(a.B, l.total + dim, cs2d_bwd_scratch_bytes_dir(&p, &o), true);   // the parameter gradients, then dw
    g.dw = part_of(buf.params, l.total, w.sizes());
    param_views(g, buf.params, l, dim, n);
    Tensor du = merged_image(a.u, serial);
    g.ddelta = at::empty(a.delta.sizes(), a.delta.options());
    o.merge_dw = fp(g.dw);
    raise_on(cs2d_bwd_dir(&p, &o, dy.const_data_ptr(), dy.stride(0), dy.stride(1), dy.stride(2), state.const_data_ptr(), buf.scratch_ptr,
                          du.data_ptr(), g.ddelta.data_ptr(), fp(g.dA), buf.dB, buf.dC, fp(g.dD), fp(g.dbias), fp(g.ddecay),
                          stream_of(a.u)), "backward");
    g.du = du.scalar_type() == a.u.scalar_type() ? du : du.to(a.u.scalar_type());
    buf.result(a.B, g.dB, g.dC);
    if (g.dw.scalar_type() != w.scalar_type()) g.dw = g.dw.to(w.scalar_type());
    return g;
}

bool wants_grad(const Tensor &t) { return given(t) && t.requires_grad(); }
bool any_grad(const Args &a) {
    return at::GradMode::is_enabled() && (wants_grad(a.u) || wants_grad(a.delta) || wants_grad(a.A) || wants_grad(a.B) || wants_grad(a.C) ||
                                          wants_grad(a.D) || wants_grad(a.bias) || wants_grad(a.decay));
}

// ---- autograd nodes ----------------------------------------------------------------------------------
struct ScanFunction : torch::autograd::Function<ScanFunction> {
    static Tensor forward(AutogradContext *ctx, const Tensor &u, const Tensor &delta, const Tensor &A, const Tensor &B, const Tensor &C,
                          const OptT &D, const OptT &bias, const OptT &decay, bool softplus, bool out_float) {
        at::AutoDispatchBelowADInplaceOrView below;
        auto r = scan_forward(Args{u, delta, A, B, C, opt(D), opt(bias), opt(decay), softplus}, out_float, true, deterministic_mode());
        ctx->saved_data["softplus"] = softplus;
        ctx->save_for_backward({u, delta, A, B, C, opt(D), opt(bias), opt(decay), r.second});
        return r.first;
    }
    static variable_list backward(AutogradContext *ctx, variable_list go) {
        const auto s = ctx->get_saved_variables();
        at::NoGradGuard no_grad;
        if (!go[0].defined()) return variable_list(10);
        const Tensor dout = go[0].stride(-1) == 1 ? go[0] : go[0].contiguous();
        const Grads g = scan_backward(Args{s[0], s[1], s[2], s[3], s[4], s[5], s[6], s[7], ctx->saved_data["softplus"].toBool()}, dout, s[8],
                                      std::nullopt, deterministic_mode());
        return {g.du, g.ddelta, g.dA, g.dB, g.dC, g.dD, g.dbias, g.ddecay, Tensor(), Tensor()};
    }
};

struct CrossFunction : torch::autograd::Function<CrossFunction> {
    static Tensor forward(AutogradContext *ctx, const Tensor &u_, const Tensor &delta_, const Tensor &A, const Tensor &B, const Tensor &C,
                          const Tensor &w, const OptT &D, const OptT &bias, const OptT &decay, bool softplus, bool serial) {
        at::AutoDispatchBelowADInplaceOrView below;
        const Tensor u = u_.contiguous(), delta = delta_.contiguous();   // B, C may be strided views (innermost stride 1)
        const Args a{u, delta, A, B, C, opt(D), opt(bias), opt(decay), softplus};
        cross_check(a, w);
        auto r = cross_forward(a, w, serial, true);
        ctx->saved_data["softplus"] = softplus;
        ctx->saved_data["serial"] = serial;
        ctx->save_for_backward({u, delta, A, B, C, a.D, a.bias, a.decay, w, r.second});
        return r.first.scalar_type() == u.scalar_type() ? r.first : r.first.to(u.scalar_type());
    }
    static variable_list backward(AutogradContext *ctx, variable_list go) {
        const auto s = ctx->get_saved_variables();
        at::NoGradGuard no_grad;
        if (!go[0].defined()) return variable_list(11);
        const Tensor dy = go[0].stride(-1) == 1 ? go[0] : go[0].contiguous();
        const Grads g = cross_backward(Args{s[0], s[1], s[2], s[3], s[4], s[5], s[6], s[7], ctx->saved_data["softplus"].toBool()}, s[8], dy,
                                       s[9], ctx->saved_data["serial"].toBool());
        return {g.du, g.ddelta, g.dA, g.dB, g.dC, g.dw, g.dD, g.dbias, g.ddecay, Tensor(), Tensor()};
    }
};

// The problem as the bytes of a cs2d_problem, for the callers that own their buffers
py::bytes py_problem(const Tensor &u, const Tensor &delta, const Tensor &A, const Tensor &B, const Tensor &C, const OptT &D, const OptT &bias,
                     const OptT &decay, bool softplus, at::ScalarType out_type, const std::string &who, bool shared_u) {
    const cs2d_problem p = make_problem(Args{u, delta, A, B, C, opt(D), opt(bias), opt(decay), softplus}, out_type, who.c_str(), shared_u);
    return py::bytes(reinterpret_cast<const char *>(&p), sizeof(p));
}

// ---- Python entry points -----------------------------------------------------------------------------
Args args_of(const Tensor &u, const Tensor &delta, const Tensor &A, const Tensor &B, const Tensor &C, const OptT &D, const OptT &bias,
             bool softplus, const OptT &decay) {
    return Args{u, delta, A, B, C, opt(D), opt(bias), opt(decay), softplus};
}

std::vector<Tensor> py_fwd(const Tensor &u, const Tensor &delta, const Tensor &A, const Tensor &B, const Tensor &C, const OptT &D,
                           const OptT &bias, bool softplus, bool out_float, const OptT &decay, const std::optional<bool> &deterministic) {
    at::NoGradGuard no_grad;
    auto r = scan_forward(args_of(u, delta, A, B, C, D, bias, softplus, decay), out_float, true, deterministic.value_or(deterministic_mode()));
    return {r.first, f32(u, 0), r.second, f32(u, 0)};
}
Tensor py_fwd_only(const Tensor &u, const Tensor &delta, const Tensor &A, const Tensor &B, const Tensor &C, const OptT &D,
                   const OptT &bias, bool softplus, bool out_float, const OptT &decay) {
    at::NoGradGuard no_grad;
    return scan_forward(args_of(u, delta, A, B, C, D, bias, softplus, decay), out_float, false, false).first;
}
std::vector<OptT> py_bwd(const Tensor &u, const Tensor &delta, const Tensor &A, const Tensor &B, const Tensor &C, const OptT &D,
                         const OptT &bias, const Tensor &dout, const OptT &state, bool softplus, const OptT &decay,
                         const OptT &param_grads, const std::optional<bool> &deterministic) {
    at::NoGradGuard no_grad;
    const Grads g = scan_backward(args_of(u, delta, A, B, C, D, bias, softplus, decay), dout, opt(state), param_grads,
                                  deterministic.value_or(deterministic_mode()));
    std::vector<OptT> r;
    for (const Tensor &t : {g.du, g.ddelta, g.dA, g.dB, g.dC, g.dD, g.dbias, g.ddecay}) r.push_back(given(t) ? OptT(t) : OptT());
    return r;
}
Tensor py_scan(const Tensor &u, const Tensor &delta, const Tensor &A, const Tensor &B, const Tensor &C, const OptT &D, const OptT &bias,
               bool softplus, bool out_float, const OptT &decay) {
    const Args a = args_of(u, delta, A, B, C, D, bias, softplus, decay);
    if (!any_grad(a)) return scan_forward(a, out_float, false, false).first;   // nothing can ask for a gradient: no saved state
    return ScanFunction::apply(u, delta, A, B, C, D, bias, decay, softplus, out_float);
}
Tensor py_cross(const Tensor &u, const Tensor &delta, const Tensor &A, const Tensor &B, const Tensor &C, const Tensor &w, const OptT &D,
                const OptT &bias, bool softplus, const OptT &decay, const std::optional<bool> &deterministic) {
    Args a = args_of(u, delta, A, B, C, D, bias, softplus, decay);
    const bool serial = deterministic.value_or(deterministic_mode());
    if (any_grad(a) || (at::GradMode::is_enabled() && w.requires_grad()))
        return CrossFunction::apply(u, delta, A, B, C, w, D, bias, decay, softplus, serial);
    cross_check(a, w);   // evaluation: no saved state
    at::NoGradGuard no_grad;
    a.u = u.contiguous(); a.delta = delta.contiguous();
    const Tensor y = cross_forward(a, w, serial, false).first;
    return y.scalar_type() == u.scalar_type() ? y : y.to(u.scalar_type());
}

// the two halves of the four-corner operator on their own: (y fp32, state), then the gradients
std::tuple<Tensor, OptT> py_cross_fwd(const Tensor &u, const Tensor &delta, const Tensor &A, const Tensor &B, const Tensor &C, const Tensor &w,
                                      const OptT &D, const OptT &bias, bool softplus, bool keep_state, const OptT &decay, bool serial) {
    at::NoGradGuard no_grad;
    const Args a = args_of(u, delta, A, B, C, D, bias, softplus, decay);
    cross_check(a, w);
    auto r = cross_forward(a, w, serial, keep_state);
    return {r.first, keep_state ? OptT(r.second) : OptT()};
}
std::vector<OptT> py_cross_bwd(const Tensor &u, const Tensor &delta, const Tensor &A, const Tensor &B, const Tensor &C, const Tensor &w,
                               const OptT &D, const OptT &bias, const Tensor &dy, const Tensor &state, bool softplus, const OptT &decay,
                               bool serial) {
    at::NoGradGuard no_grad;
    const Args a = args_of(u, delta, A, B, C, D, bias, softplus, decay);
    cross_check(a, w);
    const Grads g = cross_backward(a, w, dy, state, serial);
    std::vector<OptT> r;
    for (const Tensor &t : {g.du, g.ddelta, g.dA, g.dB, g.dC, g.dw, g.dD, g.dbias, g.ddecay}) r.push_back(given(t) ? OptT(t) : OptT());
    return r;
}

}  // namespace

PYBIND11_MODULE(_native, m) {
    m.doc() = "native host path of the cs2d operators (see cs2d/ops.py and cs2d/cross.py)";
    m.def("problem", &py_problem);
    m.def("fwd", &py_fwd, py::call_guard<py::gil_scoped_release>());
    m.def("fwd_only", &py_fwd_only, py::call_guard<py::gil_scoped_release>());
    m.def("bwd", &py_bwd, py::call_guard<py::gil_scoped_release>());
    m.def("scan", &py_scan, py::call_guard<py::gil_scoped_release>());
    m.def("cross", &py_cross, py::call_guard<py::gil_scoped_release>());
    m.def("cross_fwd", &py_cross_fwd, py::call_guard<py::gil_scoped_release>());
    m.def("cross_bwd", &py_cross_bwd, py::call_guard<py::gil_scoped_release>());
}
