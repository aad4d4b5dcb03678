// PyTorch binding of the WKV ops: argument checks, output and workspace allocation, autograd nodes.
// All of it is host work on the way to the C ABI; it is native because a call of the op is a handful of
// microsecond kernels when heads, tokens or batch are few, and the same steps in Python take hundreds of
// microseconds (v6, 5 heads, 4096-token segments: 284 us per call in Python, of which the GPU was busy 56).
#include "native_ops.h"

namespace wkv_native {

// ------------------------------------------------------------------------------ status words
namespace {
constexpr int MAX_DEVICES = 64;
std::atomic<int *> g_status[MAX_DEVICES];
std::mutex g_status_lock;

void raise_if_set(int device, int *word) {
    if (__atomic_load_n(word, __ATOMIC_ACQUIRE) == 0) return;
    // reported once; taken and cleared in one step, so that a bit a kernel sets meanwhile is reported by this look or the next
    const int code = __atomic_exchange_n(word, 0, __ATOMIC_ACQ_REL);
    if (code == 0) return;      // (another thread reports it)
    TORCH_CHECK(false, "a v5/v6 call on cuda:", device, ": a device-side wait ran out (status ", code,
                "); the outputs of that call are invalid");
}
}  // namespace

int *status_word(int device) {
    TORCH_CHECK(device >= 0 && device < MAX_DEVICES, "device index out of range");
    int *p = g_status[device].load(std::memory_order_acquire);
    if (p == nullptr) {
        std::lock_guard<std::mutex> hold(g_status_lock);
        p = g_status[device].load(std::memory_order_acquire);
        if (p == nullptr) {
            // a cache line per device, kept for the life of the process
            C10_CUDA_CHECK(cudaHostAlloc((void **)&p, 128, cudaHostAllocPortable | cudaHostAllocMapped));
            *p = 0;
            g_status[device].store(p, std::memory_order_release);
        }
    }
    return p;
}

void poll_status(int device, bool wait) {
    for (int d = 0; d < MAX_DEVICES; d++) {
        int *p = g_status[d].load(std::memory_order_acquire);
        if ((device >= 0 && d != device) || p == nullptr) continue;
        if (wait) {
            c10::cuda::CUDAGuard guard(d);
            C10_CUDA_CHECK(cudaDeviceSynchronize());
        }
        raise_if_set(d, p);
    }
}

// ------------------------------------------------------------------------------ v5 / v6 calls
namespace {

wkv_args_t make_args(const Tensor &r, int w_kind, int layout, int path, int time_groups) {
    wkv_args_t a = {};
    a.B = (int)r.size(0); a.T = (int)r.size(1); a.H = (int)(r.size(2) / HEAD); a.N = (int)HEAD;
    a.dtype = dtype_code(r.scalar_type());
    a.w_kind = w_kind; a.state_layout = layout; a.path = path; a.time_groups = time_groups;
    return a;
}

void check_btc(const Tensor &r, const Tensor &t, const char *name) {
    TORCH_CHECK_VALUE(t.sizes() == r.sizes(), name, " must have shape ", r.sizes(), ", got ", t.sizes());
    TORCH_CHECK_VALUE(t.is_contiguous(), name, " must be contiguous (a [:, t0:t1] view of a longer tensor is not)");
}
// a parameter or a state: `n` elements of type `dt`
void check_flat(const Tensor &t, int64_t n, at::ScalarType dt, const char *name) {
    if (!t.defined()) return;
    TORCH_CHECK_VALUE(t.numel() == n, name, " must have ", n, " elements, got ", t.sizes());
    TORCH_CHECK_VALUE(t.scalar_type() == dt, name, " must be ", dt, ", got ", t.scalar_type());
    TORCH_CHECK_VALUE(t.is_contiguous(), name, " must be contiguous");
}
// the kernels take raw pointers: everything has to have the element type and size they assume
void check_call(bool v6, const Tensor &r, const Tensor &k, const Tensor &v, const Tensor &w, const Tensor &u,
                const Tensor &state, int w_kind) {
    TORCH_CHECK_VALUE(r.dim() == 3 && r.size(2) % HEAD == 0, "r must be [B,T,H*64]");
    const auto dt = r.scalar_type();
    check_btc(r, r, "r"); check_btc(r, k, "k"); check_btc(r, v, "v");
    if (v6) check_btc(r, w, "w");
    check_flat(k, r.numel(), dt, "k"); check_flat(v, r.numel(), dt, "v");
    check_flat(w, v6 ? r.numel() : r.size(2), v6 && w_kind == WKV_W_RAW ? dt : at::kFloat, "w");
    check_flat(u, r.size(2), dt, "u");
    check_flat(state, r.size(0) * r.size(2) * HEAD, at::kFloat, "the state");
}

}  // namespace

Fwd wkv56_forward(bool v6, const Tensor &r, const Tensor &k, const Tensor &v, const Tensor &w, const Tensor &u,
                  const Tensor &state_in, int w_kind, int layout, int path, const Tensor &state_out, bool save_ckpt,
                  int time_groups, const Tensor &saved, int saved_mode, bool sync_check) {
    check_call(v6, r, k, v, w, u, state_in, w_kind);
    require_cuda({&r, &k, &v, &w, &u, &state_in, &state_out});
    check_flat(state_out, r.size(0) * r.size(2) * HEAD, at::kFloat, "state_out");
    const int dev = r.device().index();
    int *status = status_word(dev);
    raise_if_set(dev, status);
    c10::cuda::OptionalCUDAGuard guard(r.device());
    Fwd out;
    out.y = fresh_like(r);
    wkv_args_t a = make_args(r, w_kind, layout, path, time_groups);
    out.state_out = state_out.defined() ? state_out : fresh({a.B, a.H, HEAD, HEAD}, at::kFloat, r);
    a.r = ptr(r); a.k = ptr(k); a.v = ptr(v); a.w = ptr(w); a.u = ptr(u);
    a.state_in = (const float *)ptr(state_in);
    a.y = ptr(out.y); a.state_out = (float *)ptr(out.state_out);
    if (save_ckpt) {
        a.state_ckpt_bytes = wkv56_state_ckpt_bytes(&a, v6);
        out.ckpt = bytes_like(r, a.state_ckpt_bytes);
        a.state_ckpt = ptr(out.ckpt);
    }
    if (saved_mode != WKV_GROUP_STATES_NONE) {
        a.group_states = ptr(saved);
        a.group_states_bytes = (size_t)saved.numel();
        a.group_states_mode = saved_mode;
    }
    a.workspace_bytes = v6 ? wkv6_forward_workspace(&a) : wkv5_forward_workspace(&a);
    Tensor ws = bytes_like(r, a.workspace_bytes);
    a.workspace = ptr(ws);
    check(wkv56x_forward(&a, v6, status, stream_of(r)), v6 ? "wkv6_forward" : "wkv5_forward");
    if (sync_check) poll_status(dev, true);
    return out;
}

Bwd wkv56_backward(bool v6, const Tensor &r, const Tensor &k, const Tensor &v, const Tensor &w, const Tensor &u,
                   const Tensor &state_in, const Tensor &gy, const Tensor &gstate_out, int w_kind, int layout, int path,
                   bool want_gstate, const Tensor &ckpt, int time_groups, bool per_batch, at::ScalarType u_type,
                   at::ScalarType w_type, bool sync_check) {
    check_call(v6, r, k, v, w, u, state_in, w_kind);
    require_cuda({&r, &k, &v, &w, &u, &state_in, &gy, &gstate_out});
    check_btc(r, gy, "gy");
    check_flat(gy, r.numel(), r.scalar_type(), "gy");
    check_flat(gstate_out, r.size(0) * r.size(2) * HEAD, at::kFloat, "gstate_out");
    const int dev = r.device().index();
    int *status = status_word(dev);
    raise_if_set(dev, status);
    c10::cuda::OptionalCUDAGuard guard(r.device());
    wkv_args_t a = make_args(r, w_kind, layout, path, time_groups);
    const int64_t B = a.B, H = a.H;
    Bwd g;
    g.gr = fresh_like(r); g.gk = fresh_like(r); g.gv = fresh_like(r);
    const bool empty = B == 0 || H == 0;
    if (per_batch) {
        g.gu = fresh({B, H * HEAD}, at::kFloat, r);
        g.gw = v6 ? fresh_like(r) : fresh({B, H * HEAD}, at::kFloat, r);
    } else {
        g.gu = empty ? at::zeros({H, HEAD}, r.options().dtype(u_type)) : fresh({H, HEAD}, u_type, r);
        g.gw = v6 ? fresh_like(r)
                  : (empty ? at::zeros({H, HEAD}, r.options().dtype(w_type)) : fresh({H, HEAD}, w_type, r));
    }
    if (want_gstate) g.gstate_in = fresh({B, H, HEAD, HEAD}, at::kFloat, r);
    a.r = ptr(r); a.k = ptr(k); a.v = ptr(v); a.w = ptr(w); a.u = ptr(u);
    a.state_in = (const float *)ptr(state_in);
    a.gy = ptr(gy); a.gstate_out = (const float *)ptr(gstate_out);
    a.gr = ptr(g.gr); a.gk = ptr(g.gk); a.gv = ptr(g.gv);
    if (v6 || per_batch) a.gw = ptr(g.gw);
    if (per_batch) a.gu = (float *)ptr(g.gu);
    a.gstate_in = (float *)ptr(g.gstate_in);
    if (ckpt.defined()) { a.state_ckpt = ptr(ckpt); a.state_ckpt_bytes = (size_t)ckpt.numel(); }
    const char *what = v6 ? "wkv6_backward" : "wkv5_backward";
    a.workspace_bytes = !per_batch ? wkv56x_backward_workspace(&a, v6)
                                   : (v6 ? wkv6_backward_workspace(&a) : wkv5_backward_workspace(&a));
    Tensor ws = bytes_like(r, a.workspace_bytes);
    a.workspace = ptr(ws);
    if (per_batch) {
        // (the public entry point keeps its status word in the workspace: read it there when asked to)
        check((v6 ? wkv6_backward : wkv5_backward)(&a, stream_of(r)), what);
        if (sync_check && ws.defined() && wkv56_uses_chunked(&a, v6)) {
            const int code = ws.slice(0, 0, 4).view(at::kInt).item<int>();
            TORCH_CHECK(code == 0, what, ": a device-side wait ran out (status ", code, ")");
        }
    } else {
        check(wkv56x_backward(&a, v6, status, ptr(g.gu), dtype_code(u_type), v6 ? nullptr : ptr(g.gw),
                              v6 ? 0 : dtype_code(w_type), stream_of(r)),
              what);
        if (sync_check) poll_status(dev, true);
    }
    return g;
}

// ------------------------------------------------------------------------------ v5 / v6 autograd node
namespace {

struct Wkv56Backward : OpNode {
    bool v6, sync;
    int path;
    at::ScalarType k_type, v_type, w_type, u_type, s_type;      // of the caller's tensors
    std::vector<int64_t> w_shape, u_shape, s_shape;
    std::string name() const override { return "Wkv56Backward"; }
    variable_list apply(variable_list &&grads) override {
        at::AutoDispatchBelowADInplaceOrView below;
        const variable_list st = unpack();
        const Tensor &r = st[0];
        const Tensor gy = grads[0].defined() ? as_contig(grads[0], r.scalar_type()) : at::zeros_like(r);
        const Tensor gs = grads[1].defined() ? as_contig(grads[1], at::kFloat) : Tensor();
        Bwd g = wkv56_backward(v6, r, st[1], st[2], st[3], st[4], st[5], gy, gs, WKV_W_RAW, WKV_STATE_KV, path, task_should_compute_output(5),
                               st[6], 0, false, abi_type(u_type), abi_type(w_type), sync);
        return {g.gr, as_input(g.gk, k_type, g.gk.sizes()), as_input(g.gv, v_type, g.gv.sizes()), as_input(g.gw, w_type, w_shape),
                as_input(g.gu, u_type, u_shape), as_input(g.gstate_in, s_type, s_shape)};
    }
};

void check_shapes56(bool v6, int64_t B, int64_t T, int64_t C, int64_t H, const Tensor &r, const Tensor &k, const Tensor &v,
                    const Tensor &w, const Tensor &u, const Tensor &state) {
    TORCH_CHECK_VALUE(C == H * HEAD, "C must equal H*64");
    const auto is_btc = [&](const Tensor &t) { return t.dim() == 3 && t.size(0) == B && t.size(1) == T && t.size(2) == C; };
    TORCH_CHECK_VALUE(is_btc(r), "r must be [B,T,C]");
    TORCH_CHECK_VALUE(is_btc(k), "k must be [B,T,C]");
    TORCH_CHECK_VALUE(is_btc(v), "v must be [B,T,C]");
    TORCH_CHECK_VALUE(v6 ? is_btc(w) : w.numel() == C, v6 ? "w must be [B,T,C]" : "w must have H*64 elements");
    TORCH_CHECK_VALUE(u.numel() == C, "u must have H*64 elements");
    TORCH_CHECK_VALUE(state.numel() == B * H * HEAD * HEAD, "state must be [B,H,64,64]");
}

}  // namespace

// WKV5.apply / WKV6.apply -> (y, state_out)
std::tuple<Tensor, Tensor> wkv56_apply(bool v6, int64_t B, int64_t T, int64_t C, int64_t H, const Tensor &r, const Tensor &k,
                                       const Tensor &v, const Tensor &w, const Tensor &u, const Tensor &state, int64_t path,
                                       const OptTensor &saved, int64_t saved_mode, bool sync_check) {
    check_shapes56(v6, B, T, C, H, r, k, v, w, u, state);
    const Tensor buf = saved.has_value() ? *saved : Tensor();
    if (wants_grad({&r, &k, &v, &w, &u, &state})) {
        auto node = make_node<Wkv56Backward>({r, k, v, w, u, state});
        node->v6 = v6; node->sync = sync_check; node->path = (int)path;
        node->k_type = k.scalar_type(); node->v_type = v.scalar_type(); node->w_type = w.scalar_type();
        node->u_type = u.scalar_type(); node->s_type = state.scalar_type();
        node->w_shape = w.sizes().vec(); node->u_shape = u.sizes().vec(); node->s_shape = state.sizes().vec();
        Fwd o;
        {
            at::AutoDispatchBelowADInplaceOrView below;
            const auto dt = r.scalar_type();
            const Tensor rc = contig(r), kc = as_contig(k, dt), vc = as_contig(v, dt), wc = as_contig(w, v6 ? dt : at::kFloat),
                         uc = as_contig(u, dt), sc = as_contig(state, at::kFloat);
            o = wkv56_forward(v6, rc, kc, vc, wc, uc, sc, WKV_W_RAW, WKV_STATE_KV, (int)path, Tensor(), true, 0, buf, (int)saved_mode, sync_check);
            node->keep({rc, kc, vc, wc, uc, sc, o.ckpt});
        }
        torch::autograd::set_history(o.y, node);
        torch::autograd::set_history(o.state_out, node);
        return {o.y, o.state_out};
    }
    const auto dt = r.scalar_type();
    Fwd o = wkv56_forward(v6, contig(r), as_contig(k, dt), as_contig(v, dt), as_contig(w, v6 ? dt : at::kFloat),
                          as_contig(u, dt), as_contig(state, at::kFloat), WKV_W_RAW, WKV_STATE_KV, (int)path, Tensor(), false, 0,
                          buf, (int)saved_mode, sync_check);
    return {o.y, o.state_out};
}

// ------------------------------------------------------------------------------ drop-in wrappers
// RWKV-v5/src/module/TimeMix.py:20-143 and RWKV-v6/src/module/TimeMix.py:19-109: the state is updated in
// place in the [value,key] layout and the gradient of the state after the call is taken as zero.
namespace {

struct DropinBackward : OpNode {
    bool v6, sync;
    at::ScalarType w_type, s_type;
    std::vector<int64_t> w_shape, u_shape, s_shape;
    std::string name() const override { return "WkvDropinBackward"; }
    variable_list apply(variable_list &&grads) override {
        if (!grads[0].defined()) return variable_list(6);
        at::AutoDispatchBelowADInplaceOrView below;
        const variable_list st = unpack();
        const Tensor &r = st[0];
        // (the v5 wrapper gives its state no gradient)
        const bool want_gs = v6 && task_should_compute_output(5);
        Bwd g = wkv56_backward(v6, r, st[1], st[2], st[3], st[4], st[5], as_contig(grads[0], r.scalar_type()), Tensor(), WKV_W_RAW,
                               WKV_STATE_VK, WKV_PATH_AUTO, want_gs, st[6], 0, false, r.scalar_type(), w_type, sync);
        return {g.gr, g.gk, g.gv, as_input(g.gw, w_type, w_shape), as_input(g.gu, r.scalar_type(), u_shape), as_input(g.gstate_in, s_type, s_shape)};
    }
};

}  // namespace

Tensor wkv56_dropin(bool v6, int64_t B, int64_t T, int64_t C, int64_t H, const Tensor &r, const Tensor &k, const Tensor &v,
                    const Tensor &w, const Tensor &u, const Tensor &state, bool sync_check) {
    for (const Tensor *t : {&r, &k, &v, &w, &u, &state}) TORCH_CHECK_VALUE(t->is_contiguous(), "inputs must be contiguous");
    const auto dt = r.scalar_type();
    TORCH_CHECK_TYPE(dt == k.scalar_type() && dt == v.scalar_type() && dt == u.scalar_type(), "r,k,v,u must share one dtype");
    if (!v6)
        TORCH_CHECK_TYPE(state.scalar_type() == at::kFloat && w.scalar_type() == at::kFloat, "state and w must be float32");
    dtype_code(dt);
    check_shapes56(v6, B, T, C, H, r, k, v, w, u, state);
    const bool save = wants_grad({&r, &k, &v, &w, &u, &state});
    std::shared_ptr<DropinBackward> node;
    if (save) {
        node = make_node<DropinBackward>({r, k, v, w, u, state});
        node->v6 = v6; node->sync = sync_check;
        node->w_type = w.scalar_type(); node->s_type = state.scalar_type();
        node->w_shape = w.sizes().vec(); node->u_shape = u.sizes().vec(); node->s_shape = state.sizes().vec();
    }
    Tensor y;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        const Tensor wc = as_contig(w, v6 ? dt : at::kFloat), s32 = as_contig(state, at::kFloat);
        // the chunked kernels hand the states over; the token-serial ones start backward from the state itself
        const wkv_args_t a = make_args(r, WKV_W_RAW, WKV_STATE_VK, WKV_PATH_AUTO, 0);
        const Tensor s_in = save && !wkv56_uses_chunked(&a, v6) ? s32.clone() : Tensor();
        Fwd o = wkv56_forward(v6, r, k, v, wc, u, s32, WKV_W_RAW, WKV_STATE_VK, WKV_PATH_AUTO, s32, save, 0, Tensor(),
                              WKV_GROUP_STATES_NONE, sync_check);
        if (s32.data_ptr() != state.data_ptr()) {
            Tensor dst = state.detach();
            dst.copy_(s32.view_as(state));
        }
        y = o.y;
        if (save) node->keep({r, k, v, wc, u, s_in, o.ckpt});
    }
    if (save) torch::autograd::set_history(y, node);
    return y;
}

// ------------------------------------------------------------------------------ v4
namespace {
void check_wkv4(const Tensor &w, const Tensor &u, const Tensor &k, const Tensor &v, const Tensor &state) {
    TORCH_CHECK_VALUE(k.dim() == 3, "k must be [B,T,C]");
    const int64_t C = k.size(2);
    TORCH_CHECK_VALUE(w.dim() == 1 && w.size(0) == C && u.dim() == 1 && u.size(0) == C, "time_decay and time_first must be [C]");
    TORCH_CHECK_VALUE(v.sizes() == k.sizes(), "v must match k");
    TORCH_CHECK_VALUE(state.dim() == 3 && state.size(0) == k.size(0) && state.size(1) == C && state.size(2) == 3,
                      "last_state must be [B,C,3]");
}
}  // namespace

Fwd4 wkv4_forward(const Tensor &w, const Tensor &u, const Tensor &k, const Tensor &v, const Tensor &state, bool save) {
    check_wkv4(w, u, k, v, state);
    const int B = (int)k.size(0), T = (int)k.size(1), C = (int)k.size(2);
    c10::cuda::OptionalCUDAGuard guard(k.device());
    Fwd4 o;
    o.y = fresh_like(k);
    o.state_out = fresh_like(state);
    o.ckpt = bytes_like(k, save ? wkv4_state_ckpt_bytes(B, T, C) : 0);
    check(wkv4x_forward(B, T, C, dtype_code(k.scalar_type()), ptr(w), dtype_code(w.scalar_type()), ptr(u), ptr(k), ptr(v),
                        (const float *)ptr(state), ptr(o.y), (float *)ptr(o.state_out), ptr(o.ckpt), stream_of(k)),
          "wkv4_forward");
    return o;
}

Bwd4 wkv4_backward(const Tensor &w, const Tensor &u, const Tensor &k, const Tensor &v, const Tensor &state, const Tensor &ckpt,
                   const Tensor &gy, const Tensor &gstate_out, at::ScalarType u_type, bool want_gstate) {
    const int B = (int)k.size(0), T = (int)k.size(1), C = (int)k.size(2);
    c10::cuda::OptionalCUDAGuard guard(k.device());
    Bwd4 g;
    g.gw = B ? fresh_like(w) : at::zeros_like(w);
    g.gu = B ? fresh({C}, u_type, u) : at::zeros({C}, u.options().dtype(u_type));
    g.gk = fresh_like(k);
    g.gv = fresh_like(v);
    if (want_gstate) g.gstate = fresh_like(state);
    Tensor ws = bytes_like(k, wkv4x_backward_workspace(B, T, C, ckpt.defined()));
    check(wkv4x_backward(B, T, C, dtype_code(k.scalar_type()), ptr(w), dtype_code(w.scalar_type()), ptr(u), ptr(k), ptr(v),
                         (const float *)ptr(state), ptr(gy), (const float *)ptr(gstate_out), ptr(g.gw), ptr(g.gu), dtype_code(u_type),
                         ptr(g.gk), ptr(g.gv), (float *)ptr(g.gstate), ptr(ws), ptr(ckpt), stream_of(k)),
          "wkv4_backward");
    return g;
}

namespace {

// RWKV-v4neo/cuda/wkv_op_bf16.cpp:13-92
struct Wkv4Backward : OpNode {
    at::ScalarType w_type, u_type, v_type, s_type;
    std::string name() const override { return "Wkv4Backward"; }
    variable_list apply(variable_list &&grads) override {
        at::AutoDispatchBelowADInplaceOrView below;
        const variable_list st = unpack();
        const Tensor &k = st[2];
        const Tensor gy = grads[0].defined() ? as_contig(grads[0], k.scalar_type()) : at::zeros_like(k);
        const Tensor gs = grads[1].defined() ? as_contig(grads[1], at::kFloat) : Tensor();
        Bwd4 g = wkv4_backward(st[0], st[1], k, st[3], st[4], st[5], gy, gs, abi_type(u_type),
                               task_should_compute_output(4));
        return {as_input(g.gw, w_type, g.gw.sizes()), as_input(g.gu, u_type, g.gu.sizes()), g.gk, as_input(g.gv, v_type, g.gv.sizes()),
                as_input(g.gstate, s_type, st[4].sizes())};
    }
};

}  // namespace

std::vector<Tensor> wkv4(const Tensor &w, const Tensor &u, const Tensor &k, const Tensor &v, const Tensor &state) {
    check_wkv4(w, u, k, v, state);
    require_cuda({&w, &u, &k, &v, &state});
    dtype_code(k.scalar_type());
    const bool save = wants_grad({&w, &u, &k, &v, &state});
    std::shared_ptr<Wkv4Backward> node;
    if (save) {
        node = make_node<Wkv4Backward>({w, u, k, v, state});
        node->w_type = w.scalar_type(); node->u_type = u.scalar_type(); node->v_type = v.scalar_type(); node->s_type = state.scalar_type();
    }
    Fwd4 o;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        const auto dt = k.scalar_type();
        const Tensor wc = as_contig(w, param_type(w)), uc = as_contig(u, dt), kc = contig(k), vc = as_contig(v, dt),
                     sc = as_contig(state, at::kFloat);
        o = wkv4_forward(wc, uc, kc, vc, sc, save);
        if (save) node->keep({wc, uc, kc, vc, sc, o.ckpt});
    }
    if (save) {
        torch::autograd::set_history(o.y, node);
        torch::autograd::set_history(o.state_out, node);
    }
    return {o.y, o.state_out};
}

}  // namespace wkv_native

TORCH_LIBRARY(rwkv, m) {
    // RWKV-v4neo/cuda/wkv_op_bf16.cpp:98
    m.def("wkv(Tensor w, Tensor u, Tensor k, Tensor v, Tensor last_state) -> Tensor[]");
    m.impl("wkv", c10::DispatchKey::CompositeImplicitAutograd, TORCH_FN(wkv_native::wkv4));
}

namespace {
using namespace wkv_native;
Tensor opt(const OptTensor &t) { return t.has_value() ? *t : Tensor(); }
py::object none_or(const Tensor &t) { return t.defined() ? py::cast(t) : py::none(); }
}  // namespace

void bind_timemix(py::module_ &m);
void bind_blocks(py::module_ &m);

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.def("wkv56_apply", &wkv56_apply);
    m.def("wkv56_dropin", &wkv56_dropin);
    m.def("wkv4", &wkv4);
    m.def("poll_status", &poll_status, py::call_guard<py::gil_scoped_release>());     // (it may wait for the device)
    m.def("status_word", [](int device) { return (uintptr_t)status_word(device); });      // its address (tests)
    m.def("wkv56_forward",
          [](bool v6, const Tensor &r, const Tensor &k, const Tensor &v, const Tensor &w, const Tensor &u, const OptTensor &s,
             int w_kind, int layout, int path, const OptTensor &s_out, bool save_ckpt, int time_groups, const OptTensor &saved,
             int saved_mode, bool sync_check) {
              at::NoGradGuard no_grad;
              Fwd o = wkv56_forward(v6, r, k, v, w, u, opt(s), w_kind, layout, path, opt(s_out), save_ckpt, time_groups, opt(saved),
                                    saved_mode, sync_check);
              return py::make_tuple(o.y, o.state_out, none_or(o.ckpt));
          });
    m.def("wkv56_backward",
          [](bool v6, const Tensor &r, const Tensor &k, const Tensor &v, const Tensor &w, const Tensor &u, const OptTensor &s,
             const Tensor &gy, const OptTensor &gs, int w_kind, int layout, int path, bool want_gstate, const OptTensor &ckpt,
             int time_groups, bool sync_check) {
              at::NoGradGuard no_grad;
              Bwd g = wkv56_backward(v6, r, k, v, w, u, opt(s), gy, opt(gs), w_kind, layout, path, want_gstate, opt(ckpt), time_groups,
                                     true, at::kFloat, at::kFloat, sync_check);
              return py::make_tuple(g.gr, g.gk, g.gv, g.gw, g.gu, none_or(g.gstate_in));
          });
    bind_timemix(m);
    bind_blocks(m);
}
