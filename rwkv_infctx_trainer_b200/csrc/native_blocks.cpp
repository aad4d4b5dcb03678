// The time-mix blocks as one autograd node each: the projections are library GEMMs, everything between them is a
// kernel of libwkv_b200.so, and the whole block is one call from Python.  (As Python modules over separate
// autograd functions a block cost 1.5 ms of host time per forward and backward, six times what the GPU needed for a
// small one; and its stacked mixes and states went through cat, slice and add kernels of their own.)
//
// Numerics are those of the separate functions: bf16 tensors, fp32 inside every kernel.
#include "native_ops.h"

namespace wkv_native {
namespace {

constexpr auto BF16 = at::kBFloat16;

// a parameter as the GEMMs take it
Tensor as_bf16(const Tensor &p) { return as_contig(p, BF16); }
// x @ W^T into `out`
void linear_into(Tensor out, const Tensor &x, const Tensor &W) { at::mm_out(out, x, W.t()); }

// the parameters of a group of mixes: pointers for the kernels, in one element type
struct Mixes {
    std::vector<Tensor> t;
    at::ScalarType type;
    bool one_minus;
    Mixes(std::initializer_list<Tensor> ps, bool one_minus_) : one_minus(one_minus_) {
        type = param_type(*ps.begin());
        for (const Tensor &p : ps)
            if (param_type(p) != type) type = at::kFloat;
        for (const Tensor &p : ps) t.push_back(as_param(p, type));
    }
    int n() const { return (int)t.size(); }
    std::array<const void *, 5> ptrs() const {
        std::array<const void *, 5> p{};
        for (int i = 0; i < n(); i++) p[i] = ptr(t[i]);
        return p;
    }
};

Tensor mix_forward(const Tensor &x, const Tensor &shift, const Mixes &mx, const Tensor &m) {
    const int B = (int)x.size(0), T = (int)x.size(1), C = (int)x.size(2);
    Tensor out = fresh({mx.n(), B * (int64_t)T, C}, x.scalar_type(), x);
    const auto p = mx.ptrs();
    check(wkvx_ddlerp_forward(B, T, C, mx.n(), ptr(x), ptr(shift), p.data(), dtype_code(mx.type), mx.one_minus, ptr(m), ptr(out), stream_of(x)),
          "wkv_ddlerp_forward");
    return out;
}

struct MixGrads {
    Tensor gx, gm, gshift;
    std::vector<Tensor> gmaa;       // in the kernel's parameter type
};
// gshift_in: gradient of the row's last token (the block's new shift state); *_add: gradients to accumulate
MixGrads mix_backward(const Tensor &x, const Tensor &shift, const Mixes &mx, const Tensor &m, const Tensor &gout,
                      const Tensor &gshift_in, const Tensor &gx_add, const Tensor &gshift_add) {
    const int B = (int)x.size(0), T = (int)x.size(1), C = (int)x.size(2);
    MixGrads g;
    g.gx = fresh_like(x);
    if (m.defined()) g.gm = fresh_like(m);
    g.gshift = fresh_like(shift);
    std::array<void *, 5> gp{};
    for (int i = 0; i < mx.n(); i++) {
        g.gmaa.push_back(fresh_like(mx.t[i]));
        gp[i] = ptr(g.gmaa[i]);
    }
    const size_t n = wkv_ddlerp_backward_workspace(B, T, C, mx.n());
    Tensor ws = bytes_like(x, n);
    const auto p = mx.ptrs();
    check(wkvx_ddlerp_backward(B, T, C, mx.n(), ptr(x), ptr(shift), p.data(), dtype_code(mx.type), mx.one_minus, ptr(m), ptr(gout),
                               ptr(gshift_in), ptr(gx_add), ptr(gshift_add), ptr(g.gx), ptr(g.gm), ptr(g.gshift), gp.data(), ptr(ws), n,
                               stream_of(x)),
          "wkv_ddlerp_backward");
    return g;
}

// GroupNorm(y) * silu(g)
Tensor norm_gate_forward(const Tensor &y, const Tensor &g, const Tensor &lw, const Tensor &lb, double eps, int64_t H) {
    Tensor out = fresh_like(y);
    check(wkvx_lnx_gate_forward((int)y.size(0), (int)H, ptr(y), ptr(g), ptr(lw), ptr(lb), dtype_code(lw.scalar_type()), (float)eps, 1, ptr(out),
                                stream_of(y)),
          "wkv_lnx_gate_forward");
    return out;
}
struct NormGrads {
    Tensor gy, gg, glw, glb;
};
NormGrads norm_gate_backward(const Tensor &y, const Tensor &g, const Tensor &lw, const Tensor &lb, double eps, int64_t H, const Tensor &gout) {
    NormGrads r{fresh_like(y), fresh_like(g), fresh_like(lw), fresh_like(lb)};
    const int tokens = (int)y.size(0);
    const size_t n = wkv_lnx_gate_backward_workspace(tokens, (int)H);
    Tensor ws = bytes_like(y, n);
    check(wkvx_lnx_gate_backward(tokens, (int)H, ptr(y), ptr(g), ptr(lw), ptr(lb), dtype_code(lw.scalar_type()), (float)eps, 1, ptr(gout),
                                 ptr(r.gy), ptr(r.gg), ptr(r.glw), ptr(r.glb), ptr(ws), n, stream_of(y)),
          "wkv_lnx_gate_backward");
    return r;
}

// Which gradients a backward pass is asked for: x, the shift state, the wkv state, then the parameters.  What nobody asks
// for is not formed -- the weight gradients of frozen projections are a third of a block's GEMM work.
struct Wanted {
    std::vector<char> w;
    bool shared(int i) const { return w[i]; }           // 0 x, 1 shift, 2 state
    bool operator()(int i) const { return w[3 + i]; }
    bool any(int first, int last) const {
        for (int i = first; i <= last; i++)
            if (w[3 + i]) return true;
        return false;
    }
};

// what every block's Function is given and keeps besides its tensors
struct Meta {
    int64_t H = 0;
    double eps = 0;
    bool sync = false;
};

Tensor last_token(const Tensor &x) { return x.select(1, x.size(1) - 1).contiguous(); }

// A forward pass of a block: with `keep` it also appends what the backward pass reads.
struct Out {
    Tensor out, shift, state;
};

// Whether decode.cu takes the call: one token of a few rows, at widths where its matrix-vector kernel beats the library's
// GEMMs.  It reads the input rows from shared memory again for every output row (1, 2, 4 or 8 of them, the next that
// holds M), so the line falls with the width.  One block of a chain over cold weights, us, decode kernels / library path,
// as a CUDA graph (called from Python the library path is 13 to 80 us longer, the decode kernels 3):
//             v6  M=1        M=2        M=4        M=8           v5  M=1        M=2        M=4        M=8
//   C = 768       19 / 49    22 / 49    24 / 49    30 / 50           10 / 33    10 / 33    12 / 32    16 / 33
//   C = 2048                            38 / 69    53 / 69                                 31 / 48    49 / 48
//   C = 2560      37 / 76    42 / 73    49 / 74    76 / 74           24 / 54    28 / 54    39 / 53    75 / 53
//   C = 4096      62 / 108   66 / 105   84 / 105   138 / 106         52 / 83    59 / 80    85 / 79    167 / 82
//   C = 6144     101 / 114  116 / 120  163 / 121   291 / 125         92 / 89   117 / 90   181 / 91    405 / 95
//   C = 8192     162 / 171  197 / 174  268 / 174                    162 / 138  202 / 138  322 / 137
// (M = 5 takes what 8 takes: the rule is by the kernels' row counts.)
bool decode_fits(const Tensor &x, int64_t att) {
    const int64_t M = x.size(0), width = std::max(x.size(2), att);
    return x.size(1) == 1 && M >= 1 && M <= wkvx_decode_max_rows() && x.size(2) % 8 == 0 && width <= (M == 1 ? 6144 : M <= 4 ? 4096 : 2048);
}

// ------------------------------------------------------------------------------ v6
// params: time_maa_x, _w, _k, _v, _r, _g, time_maa_w1, w2, time_decay, time_decay_w1, w2, time_faaaa, receptance, key, value,
// output, gate, ln_x.weight, ln_x.bias
enum { P6_X, P6_MW, P6_MK, P6_MV, P6_MR, P6_MG, P6_W1, P6_W2, P6_DECAY, P6_D1, P6_D2, P6_U, P6_R, P6_K, P6_V, P6_O, P6_G, P6_LW, P6_LB, P6_N };

Mixes first6(const variable_list &p) { return Mixes({p[P6_X]}, false); }
Mixes five6(const variable_list &p) { return Mixes({p[P6_MW], p[P6_MK], p[P6_MV], p[P6_MR], p[P6_MG]}, false); }

Out forward6(const Tensor &x, const Tensor &shift, const Tensor &state, const variable_list &p, const Meta &me, variable_list *keep) {
    const int64_t B = x.size(0), T = x.size(1), C = x.size(2), M = B * T, H = me.H;
    if (!keep && decode_fits(x, H * HEAD) && C == H * HEAD && p[P6_W2].dim() == 3 && p[P6_W2].size(1) == 32 && p[P6_D2].size(0) % 8 == 0) {
        // one token of a few rows: the block's own kernels
        const Mixes mx({p[P6_X], p[P6_MW], p[P6_MK], p[P6_MV], p[P6_MR], p[P6_MG]}, false);
        const auto lt = param_type(p[P6_LW]);
        const Tensor w1 = as_bf16(p[P6_W1]), w2 = as_bf16(p[P6_W2]), td = as_bf16(p[P6_DECAY]), d1 = as_bf16(p[P6_D1]), d2 = as_bf16(p[P6_D2]),
                     u = as_bf16(p[P6_U]), lw = as_param(p[P6_LW], lt), lb = as_param(p[P6_LB], lt);
        const Tensor proj[5] = {as_bf16(p[P6_R]), as_bf16(p[P6_K]), as_bf16(p[P6_V]), as_bf16(p[P6_G]), as_bf16(p[P6_O])};
        const int64_t R = w2.size(1), DR = d2.size(0);
        Tensor scratch = fresh({10 * M * C + M * (5 * R + DR)}, x.scalar_type(), x);
        Out o{fresh_like(x), fresh_like(shift), fresh_like(state)};
        wkvx_decode6_t a = {};
        a.M = (int)M; a.H = (int)H; a.rank = (int)R; a.decay_rank = (int)DR;
        a.x = ptr(x); a.shift = ptr(shift);
        a.maa_x = ptr(mx.t[0]);
        for (int i = 0; i < 5; i++) a.maa[i] = ptr(mx.t[1 + i]);
        a.maa_dtype = dtype_code(mx.type);
        a.w1 = ptr(w1); a.w2 = ptr(w2); a.decay = ptr(td); a.d1 = ptr(d1); a.d2 = ptr(d2); a.u = ptr(u);
        for (int i = 0; i < 5; i++) a.proj[i] = ptr(proj[i]);
        a.ln_w = ptr(lw); a.ln_b = ptr(lb); a.ln_dtype = dtype_code(lt); a.eps = (float)me.eps;
        a.state_in = (const float *)ptr(state); a.state_out = (float *)ptr(o.state);
        char *q = (char *)ptr(scratch);
        const int64_t n = M * C * 2;
        a.xs = q; a.rkvg = q + 5 * n; a.normed = q + 9 * n; a.t1 = q + 10 * n; a.dd = q + 10 * n + M * 5 * R * 2;
        a.out = ptr(o.out); a.new_shift = ptr(o.shift);
        const int err = wkvx_decode6(&a, stream_of(x));
        if (err != WKV_ERR_ALIGN) {
            check(err, "decode6");
            return o;
        }
        // (a weight that does not start on 16 bytes: the library GEMMs below take it)
    }
    // the five mixes: a first lerp feeds the low-rank map that makes them data-dependent
    const Tensor xxx = mix_forward(x, shift, first6(p), Tensor()).view({M, C});
    const Tensor w1 = as_bf16(p[P6_W1]), w2 = as_bf16(p[P6_W2]);
    const int64_t R = w2.size(1);
    Tensor t1 = at::mm(xxx, w1).tanh_();
    const Tensor m = at::bmm(t1.view({M, 5, R}).transpose(0, 1), w2);
    const Tensor xs = mix_forward(x, shift, five6(p), m);
    Tensor rkvg = fresh({4, M, C}, x.scalar_type(), x);
    linear_into(rkvg[0], xs[3], as_bf16(p[P6_R]));
    linear_into(rkvg[1], xs[1], as_bf16(p[P6_K]));
    linear_into(rkvg[2], xs[2], as_bf16(p[P6_V]));
    linear_into(rkvg[3], xs[4], as_bf16(p[P6_G]));
    Tensor dd = at::mm(xs[0], as_bf16(p[P6_D1])).tanh_();
    const Tensor w = at::addmm(as_bf16(p[P6_DECAY]).view({C}), dd, as_bf16(p[P6_D2]));
    const auto btc = [&](const Tensor &t) { return t.view({B, T, C}); };
    const Tensor u = as_bf16(p[P6_U]);
    Fwd o = wkv56_forward(true, btc(rkvg[0]), btc(rkvg[1]), btc(rkvg[2]), btc(w), u, state, WKV_W_RAW, WKV_STATE_KV, WKV_PATH_AUTO, Tensor(),
                          keep != nullptr, 0, Tensor(), WKV_GROUP_STATES_NONE, me.sync);
    const auto lt = param_type(p[P6_LW]);
    const Tensor y = o.y.view({M, C}), n = norm_gate_forward(y, rkvg[3], as_param(p[P6_LW], lt), as_param(p[P6_LB], lt), me.eps, H);
    const Tensor out = at::mm(n, as_bf16(p[P6_O]).t());
    if (keep) *keep = {xxx, t1, m, xs, rkvg, dd, w, u, y, n, o.ckpt};
    return {out.view({B, T, C}), last_token(x), o.state_out};
}

variable_list backward6(const Tensor &x, const Tensor &shift, const Tensor &state, const variable_list &p, const Meta &me,
                        const variable_list &kept, const Tensor &gout_, const Tensor &gshift_new, const Tensor &gstate, const Wanted &want) {
    const int64_t B = x.size(0), T = x.size(1), C = x.size(2), M = B * T, H = me.H;
    const Tensor &xxx = kept[0], &t1 = kept[1], &m = kept[2], &xs = kept[3], &rkvg = kept[4], &dd = kept[5], &w = kept[6], &u = kept[7],
                 &y = kept[8], &n = kept[9], &ckpt = kept[10];
    const auto btc = [&](const Tensor &t) { return t.view({B, T, C}); };
    variable_list g(3 + P6_N);
    const auto param = [&](int i) -> Tensor & { return g[3 + i]; };
    // through the low-rank map of the mixes; through the mixes; through the WKV op; through norm and gate
    const bool first = want.shared(0) || want.shared(1) || want(P6_X), mixes = first || want.any(P6_MW, P6_W2),
               wkv = mixes || want.shared(2) || want.any(P6_DECAY, P6_V), norm = wkv || want.any(P6_G, P6_LB);
    const Tensor gout = gout_.view({M, C});
    if (want(P6_O)) param(P6_O) = at::mm(gout.t(), n);
    if (!norm) return g;
    const Tensor gn = at::mm(gout, as_bf16(p[P6_O]));
    const auto lt = param_type(p[P6_LW]);
    NormGrads ng = norm_gate_backward(y, rkvg[3], as_param(p[P6_LW], lt), as_param(p[P6_LB], lt), me.eps, H, gn);
    param(P6_LW) = ng.glw;
    param(P6_LB) = ng.glb;
    if (want(P6_G)) param(P6_G) = at::mm(ng.gg.t(), xs[4]);
    if (!wkv) return g;
    Bwd o = wkv56_backward(true, btc(rkvg[0]), btc(rkvg[1]), btc(rkvg[2]), btc(w), u, state, btc(ng.gy), gstate, WKV_W_RAW, WKV_STATE_KV,
                           WKV_PATH_AUTO, want.shared(2), ckpt, 0, false, param_type(p[P6_U]), at::kFloat, me.sync);
    param(P6_U) = o.gu;
    g[2] = o.gstate_in;
    const Tensor gr = o.gr.view({M, C}), gk = o.gk.view({M, C}), gv = o.gv.view({M, C}), gw = o.gw.view({M, C});
    if (want(P6_R)) param(P6_R) = at::mm(gr.t(), xs[3]);
    if (want(P6_K)) param(P6_K) = at::mm(gk.t(), xs[1]);
    if (want(P6_V)) param(P6_V) = at::mm(gv.t(), xs[2]);
    // the decay's low-rank map
    const Tensor d1 = as_bf16(p[P6_D1]), d2 = as_bf16(p[P6_D2]);
    if (want(P6_DECAY)) param(P6_DECAY) = gw.sum(0);
    if (want(P6_D2)) param(P6_D2) = at::mm(dd.t(), gw);
    const Tensor gdd = mixes || want(P6_D1) ? at::tanh_backward(at::mm(gw, d2.t()), dd) : Tensor();
    if (want(P6_D1)) param(P6_D1) = at::mm(xs[0].t(), gdd);
    if (!mixes) return g;
    Tensor gxs = fresh_like(xs);
    const auto into = [&](int i, const Tensor &a, const Tensor &b) { Tensor d = gxs[i]; at::mm_out(d, a, b); };
    into(3, gr, as_bf16(p[P6_R]));
    into(1, gk, as_bf16(p[P6_K]));
    into(2, gv, as_bf16(p[P6_V]));
    into(4, ng.gg, as_bf16(p[P6_G]));
    into(0, gdd, d1.t());
    MixGrads mg = mix_backward(x, shift, five6(p), m, gxs, gshift_new, Tensor(), Tensor());
    for (int i = 0; i < 5; i++) param(P6_MW + i) = mg.gmaa[i];
    // the mixes' low-rank map
    const Tensor w1 = as_bf16(p[P6_W1]), w2 = as_bf16(p[P6_W2]);
    const int64_t R = w2.size(1);
    const Tensor t5 = t1.view({M, 5, R});
    if (want(P6_W2)) param(P6_W2) = at::bmm(t5.permute({1, 2, 0}), mg.gm);
    if (!first && !want(P6_W1)) return g;
    Tensor gt1 = fresh_like(t1), gt5 = gt1.view({M, 5, R});
    at::tanh_backward_out(gt5, at::bmm(mg.gm, w2.transpose(1, 2)).transpose(0, 1), t5);
    if (want(P6_W1)) param(P6_W1) = at::mm(xxx.t(), gt1);
    if (!first) return g;
    MixGrads m1 = mix_backward(x, shift, first6(p), Tensor(), at::mm(gt1, w1.t()), Tensor(), mg.gx, mg.gshift);
    param(P6_X) = m1.gmaa[0];
    g[0] = m1.gx;
    g[1] = m1.gshift;
    return g;
}

// ------------------------------------------------------------------------------ v5
// params: time_mix_k, _v, _r, _g, time_decay, time_faaaa, receptance, key, value, output, gate, ln_x.weight, ln_x.bias
enum { P5_MK, P5_MV, P5_MR, P5_MG, P5_DECAY, P5_U, P5_R, P5_K, P5_V, P5_O, P5_G, P5_LW, P5_LB, P5_N };

// x*mix + x_prev*(1-mix)  =  x + (x_prev - x)*(1-mix)
Mixes four5(const variable_list &p) { return Mixes({p[P5_MK], p[P5_MV], p[P5_MR], p[P5_MG]}, true); }

Out forward5(const Tensor &x, const Tensor &shift, const Tensor &state, const variable_list &p, const Meta &me, variable_list *keep) {
    const int64_t B = x.size(0), T = x.size(1), C = x.size(2), M = B * T, H = me.H, A = H * HEAD;
    if (!keep && decode_fits(x, A)) {
        // one token of a few rows: the block's own kernels
        const Mixes mx = four5(p);
        const auto lt = param_type(p[P5_LW]);
        const Tensor u = as_bf16(p[P5_U]), w = as_contig(p[P5_DECAY], param_type(p[P5_DECAY])), lw = as_param(p[P5_LW], lt), lb = as_param(p[P5_LB], lt);
        const Tensor proj[5] = {as_bf16(p[P5_R]), as_bf16(p[P5_K]), as_bf16(p[P5_V]), as_bf16(p[P5_G]), as_bf16(p[P5_O])};
        Tensor scratch = fresh({5 * M * A}, x.scalar_type(), x);
        Out o{fresh_like(x), fresh_like(shift), fresh_like(state)};
        wkvx_decode5_t a = {};
        a.M = (int)M; a.H = (int)H; a.C = (int)C;
        a.x = ptr(x); a.shift = ptr(shift);
        for (int i = 0; i < 4; i++) a.mix[i] = ptr(mx.t[i]);
        a.mix_dtype = dtype_code(mx.type);
        a.decay = ptr(w); a.decay_dtype = dtype_code(w.scalar_type()); a.u = ptr(u);
        for (int i = 0; i < 5; i++) a.proj[i] = ptr(proj[i]);
        a.ln_w = ptr(lw); a.ln_b = ptr(lb); a.ln_dtype = dtype_code(lt); a.eps = (float)me.eps;
        a.state_in = (const float *)ptr(state); a.state_out = (float *)ptr(o.state);
        char *q = (char *)ptr(scratch);
        a.rkvg = q; a.normed = q + 4 * M * A * 2;
        a.out = ptr(o.out); a.new_shift = ptr(o.shift);
        const int err = wkvx_decode5(&a, stream_of(x));
        if (err != WKV_ERR_ALIGN) {
            check(err, "decode5");
            return o;
        }
    }
    const Tensor xs = mix_forward(x, shift, four5(p), Tensor());
    Tensor rkvg = fresh({4, M, A}, x.scalar_type(), x);
    linear_into(rkvg[0], xs[2], as_bf16(p[P5_R]));
    linear_into(rkvg[1], xs[0], as_bf16(p[P5_K]));
    linear_into(rkvg[2], xs[1], as_bf16(p[P5_V]));
    linear_into(rkvg[3], xs[3], as_bf16(p[P5_G]));
    const auto btc = [&](const Tensor &t) { return t.view({B, T, A}); };
    const Tensor u = as_bf16(p[P5_U]), w = as_contig(p[P5_DECAY], at::kFloat);
    Fwd o = wkv56_forward(false, btc(rkvg[0]), btc(rkvg[1]), btc(rkvg[2]), w, u, state, WKV_W_RAW, WKV_STATE_KV, WKV_PATH_AUTO, Tensor(),
                          keep != nullptr, 0, Tensor(), WKV_GROUP_STATES_NONE, me.sync);
    const auto lt = param_type(p[P5_LW]);
    const Tensor y = o.y.view({M, A}), n = norm_gate_forward(y, rkvg[3], as_param(p[P5_LW], lt), as_param(p[P5_LB], lt), me.eps, H);
    const Tensor out = at::mm(n, as_bf16(p[P5_O]).t());
    if (keep) *keep = {xs, rkvg, w, u, y, n, o.ckpt};
    return {out.view({B, T, C}), last_token(x), o.state_out};
}

variable_list backward5(const Tensor &x, const Tensor &shift, const Tensor &state, const variable_list &p, const Meta &me,
                        const variable_list &kept, const Tensor &gout_, const Tensor &gshift_new, const Tensor &gstate, const Wanted &want) {
    const int64_t B = x.size(0), T = x.size(1), C = x.size(2), M = B * T, H = me.H, A = H * HEAD;
    const Tensor &xs = kept[0], &rkvg = kept[1], &w = kept[2], &u = kept[3], &y = kept[4], &n = kept[5], &ckpt = kept[6];
    const auto btc = [&](const Tensor &t) { return t.view({B, T, A}); };
    variable_list g(3 + P5_N);
    const auto param = [&](int i) -> Tensor & { return g[3 + i]; };
    const bool mixes = want.shared(0) || want.shared(1) || want.any(P5_MK, P5_MG), wkv = mixes || want.shared(2) || want.any(P5_DECAY, P5_V),
               norm = wkv || want.any(P5_G, P5_LB);
    const Tensor gout = gout_.view({M, C});
    if (want(P5_O)) param(P5_O) = at::mm(gout.t(), n);
    if (!norm) return g;
    const Tensor gn = at::mm(gout, as_bf16(p[P5_O]));
    const auto lt = param_type(p[P5_LW]);
    NormGrads ng = norm_gate_backward(y, rkvg[3], as_param(p[P5_LW], lt), as_param(p[P5_LB], lt), me.eps, H, gn);
    param(P5_LW) = ng.glw;
    param(P5_LB) = ng.glb;
    if (want(P5_G)) param(P5_G) = at::mm(ng.gg.t(), xs[3]);
    if (!wkv) return g;
    Bwd o = wkv56_backward(false, btc(rkvg[0]), btc(rkvg[1]), btc(rkvg[2]), w, u, state, btc(ng.gy), gstate, WKV_W_RAW, WKV_STATE_KV,
                           WKV_PATH_AUTO, want.shared(2), ckpt, 0, false, param_type(p[P5_U]), param_type(p[P5_DECAY]), me.sync);
    param(P5_U) = o.gu;
    param(P5_DECAY) = o.gw;
    g[2] = o.gstate_in;
    const Tensor gr = o.gr.view({M, A}), gk = o.gk.view({M, A}), gv = o.gv.view({M, A});
    if (want(P5_R)) param(P5_R) = at::mm(gr.t(), xs[2]);
    if (want(P5_K)) param(P5_K) = at::mm(gk.t(), xs[0]);
    if (want(P5_V)) param(P5_V) = at::mm(gv.t(), xs[1]);
    if (!mixes) return g;
    Tensor gxs = fresh_like(xs);
    const auto into = [&](int i, const Tensor &a, const Tensor &b) { Tensor d = gxs[i]; at::mm_out(d, a, b); };
    into(2, gr, as_bf16(p[P5_R]));
    into(0, gk, as_bf16(p[P5_K]));
    into(1, gv, as_bf16(p[P5_V]));
    into(3, ng.gg, as_bf16(p[P5_G]));
    MixGrads mg = mix_backward(x, shift, four5(p), Tensor(), gxs, gshift_new, Tensor(), Tensor());
    for (int i = 0; i < 4; i++) param(P5_MK + i) = mg.gmaa[i];
    g[0] = mg.gx;
    g[1] = mg.gshift;
    return g;
}

// ------------------------------------------------------------------------------ v4
// params: time_mix_k, _v, _r, time_decay, time_first, key, value, receptance, output
enum { P4_MK, P4_MV, P4_MR, P4_DECAY, P4_U, P4_K, P4_V, P4_R, P4_O, P4_N };

Mixes three4(const variable_list &p) { return Mixes({p[P4_MK], p[P4_MV], p[P4_MR]}, true); }

Out forward4(const Tensor &x, const Tensor &shift, const Tensor &state, const variable_list &p, const Meta &, variable_list *keep) {
    const int64_t B = x.size(0), T = x.size(1), C = x.size(2), M = B * T;
    const Tensor xs = mix_forward(x, shift, three4(p), Tensor());
    const int64_t A = p[P4_K].size(0);       // dim_att
    Tensor kv = fresh({2, M, A}, x.scalar_type(), x);
    linear_into(kv[0], xs[0], as_bf16(p[P4_K]));
    linear_into(kv[1], xs[1], as_bf16(p[P4_V]));
    Tensor sr = at::mm(xs[2], as_bf16(p[P4_R]).t()).sigmoid_();
    const Tensor w = as_contig(p[P4_DECAY], param_type(p[P4_DECAY])), u = as_bf16(p[P4_U]);
    Fwd4 o = wkv4_forward(w, u, kv[0].view({B, T, A}), kv[1].view({B, T, A}), state, keep != nullptr);
    const Tensor y = o.y.view({M, A}), sy = at::mul(sr, y), out = at::mm(sy, as_bf16(p[P4_O]).t());
    if (keep) *keep = {xs, kv, sr, w, u, y, sy, o.ckpt};
    return {out.view({B, T, C}), last_token(x), o.state_out};
}

variable_list backward4(const Tensor &x, const Tensor &shift, const Tensor &state, const variable_list &p, const Meta &,
                        const variable_list &kept, const Tensor &gout_, const Tensor &gshift_new, const Tensor &gstate, const Wanted &want) {
    const int64_t B = x.size(0), T = x.size(1), C = x.size(2), M = B * T;
    const Tensor &xs = kept[0], &kv = kept[1], &sr = kept[2], &w = kept[3], &u = kept[4], &y = kept[5], &sy = kept[6], &ckpt = kept[7];
    const int64_t A = kv.size(2);
    variable_list g(3 + P4_N);
    const auto param = [&](int i) -> Tensor & { return g[3 + i]; };
    const bool mixes = want.shared(0) || want.shared(1) || want.any(P4_MK, P4_MR), wkv = mixes || want.shared(2) || want.any(P4_DECAY, P4_V);
    const Tensor gout = gout_.view({M, C});
    if (want(P4_O)) param(P4_O) = at::mm(gout.t(), sy);
    if (!wkv && !want(P4_R)) return g;
    const Tensor gsy = at::mm(gout, as_bf16(p[P4_O])), gr = mixes || want(P4_R) ? at::sigmoid_backward(at::mul(gsy, y), sr) : Tensor();
    if (want(P4_R)) param(P4_R) = at::mm(gr.t(), xs[2]);
    if (!wkv) return g;
    Bwd4 o = wkv4_backward(w, u, kv[0].view({B, T, A}), kv[1].view({B, T, A}), state, ckpt, at::mul(gsy, sr).view({B, T, A}), gstate,
                           param_type(p[P4_U]), want.shared(2));
    param(P4_DECAY) = o.gw;
    param(P4_U) = o.gu;
    g[2] = o.gstate;
    const Tensor gk = o.gk.view({M, A}), gv = o.gv.view({M, A});
    if (want(P4_K)) param(P4_K) = at::mm(gk.t(), xs[0]);
    if (want(P4_V)) param(P4_V) = at::mm(gv.t(), xs[1]);
    if (!mixes) return g;
    Tensor gxs = fresh_like(xs);
    const auto into = [&](int i, const Tensor &a, const Tensor &b) { Tensor d = gxs[i]; at::mm_out(d, a, b); };
    into(0, gk, as_bf16(p[P4_K]));
    into(1, gv, as_bf16(p[P4_V]));
    into(2, gr, as_bf16(p[P4_R]));
    MixGrads mg = mix_backward(x, shift, three4(p), Tensor(), gxs, gshift_new, Tensor(), Tensor());
    for (int i = 0; i < 3; i++) param(P4_MK + i) = mg.gmaa[i];
    g[0] = mg.gx;
    g[1] = mg.gshift;
    return g;
}

// ------------------------------------------------------------------------------ the node
typedef Out (*ForwardFn)(const Tensor &, const Tensor &, const Tensor &, const variable_list &, const Meta &, variable_list *);
typedef variable_list (*BackwardFn)(const Tensor &, const Tensor &, const Tensor &, const variable_list &, const Meta &,
                                    const variable_list &, const Tensor &, const Tensor &, const Tensor &, const Wanted &);
typedef void (*CheckFn)(const variable_list &, int64_t C, int64_t H);
struct Kind {
    ForwardFn forward;
    BackwardFn backward;
    CheckFn check;
    size_t params;
};

// The parameters' sizes against the width of x and the head count: the kernels take pointers, and some of them run
// before (decode: instead of) any library call that would notice.
void check_vec(const Tensor &t, int64_t n, const char *name) {
    TORCH_CHECK_VALUE(t.numel() == n, name, " must have ", n, " elements for this input, got ", t.sizes());
}
void check_mat(const Tensor &t, int64_t rows, int64_t cols, const char *name) {
    TORCH_CHECK_VALUE(t.dim() == 2 && t.size(0) == rows && t.size(1) == cols, name, " must be [", rows, ",", cols, "] for this input, got ", t.sizes());
}
void check6(const variable_list &p, int64_t C, int64_t H) {
    TORCH_CHECK_VALUE(C == H * HEAD, "x must be [B,T,H*64] with H = ", H, ", got a width of ", C);
    static const char *const mixes[] = {"time_maa_x", "time_maa_w", "time_maa_k", "time_maa_v", "time_maa_r", "time_maa_g"};
    for (int i = P6_X; i <= P6_MG; i++) check_vec(p[i], C, mixes[i]);
    const Tensor &w1 = p[P6_W1], &w2 = p[P6_W2], &d1 = p[P6_D1], &d2 = p[P6_D2];
    TORCH_CHECK_VALUE(w2.dim() == 3 && w2.size(0) == 5 && w2.size(2) == C, "time_maa_w2 must be [5,rank,", C, "] for this input, got ", w2.sizes());
    check_mat(w1, C, 5 * w2.size(1), "time_maa_w1");
    check_vec(p[P6_DECAY], C, "time_decay");
    TORCH_CHECK_VALUE(d2.dim() == 2 && d2.size(1) == C, "time_decay_w2 must be [rank,", C, "] for this input, got ", d2.sizes());
    check_mat(d1, C, d2.size(0), "time_decay_w1");
    check_vec(p[P6_U], C, "time_faaaa");
    static const char *const proj[] = {"receptance", "key", "value", "output", "gate"};
    for (int i = 0; i < 5; i++) check_mat(p[P6_R + i], C, C, proj[i]);
    check_vec(p[P6_LW], C, "ln_x.weight"); check_vec(p[P6_LB], C, "ln_x.bias");
}
void check5(const variable_list &p, int64_t C, int64_t H) {
    const int64_t A = H * HEAD;
    static const char *const mixes[] = {"time_mix_k", "time_mix_v", "time_mix_r", "time_mix_g"};
    for (int i = P5_MK; i <= P5_MG; i++) check_vec(p[i], C, mixes[i]);
    check_vec(p[P5_DECAY], A, "time_decay"); check_vec(p[P5_U], A, "time_faaaa");
    check_mat(p[P5_R], A, C, "receptance"); check_mat(p[P5_K], A, C, "key"); check_mat(p[P5_V], A, C, "value"); check_mat(p[P5_G], A, C, "gate");
    check_mat(p[P5_O], C, A, "output");
    check_vec(p[P5_LW], A, "ln_x.weight"); check_vec(p[P5_LB], A, "ln_x.bias");
}
void check4(const variable_list &p, int64_t C, int64_t) {
    const int64_t A = p[P4_DECAY].numel();      // dim_att
    static const char *const mixes[] = {"time_mix_k", "time_mix_v", "time_mix_r"};
    for (int i = P4_MK; i <= P4_MR; i++) check_vec(p[i], C, mixes[i]);
    check_vec(p[P4_U], A, "time_first");
    check_mat(p[P4_K], A, C, "key"); check_mat(p[P4_V], A, C, "value"); check_mat(p[P4_R], A, C, "receptance");
    check_mat(p[P4_O], C, A, "output");
}
const Kind &kind_of(int64_t version) {
    static const Kind k4{forward4, backward4, check4, P4_N}, k5{forward5, backward5, check5, P5_N}, k6{forward6, backward6, check6, P6_N};
    TORCH_CHECK_VALUE(version >= 4 && version <= 6, "unknown block version");
    return version == 4 ? k4 : version == 5 ? k5 : k6;
}

struct BlockBackward : OpNode {
    int64_t version;
    Meta meta;
    std::string name() const override { return "TimeMixBlockBackward"; }
    variable_list apply(variable_list &&grads) override {
        at::AutoDispatchBelowADInplaceOrView below;
        const variable_list st = unpack();
        const Kind &k = kind_of(version);
        const Tensor &x = st[0], &shift = st[1], &state = st[2];
        c10::cuda::OptionalCUDAGuard guard(x.device());
        const variable_list p(st.begin() + 3, st.begin() + 3 + k.params), kept(st.begin() + 3 + k.params, st.end());
        const Tensor gout = grads[0].defined() ? as_contig(grads[0], BF16) : at::zeros_like(x);
        const Tensor gshift = grads[1].defined() ? as_contig(grads[1], BF16) : Tensor();
        const Tensor gstate = grads[2].defined() ? as_contig(grads[2], at::kFloat) : Tensor();
        Wanted want;
        for (size_t i = 0; i < 3 + k.params; i++) want.w.push_back(task_should_compute_output(i));
        variable_list g = k.backward(x, shift, state, p, meta, kept, gout, gshift, gstate, want);
        for (size_t i = 0; i < k.params; i++) g[3 + i] = as_input(g[3 + i], p[i].scalar_type(), p[i].sizes());
        return g;
    }
};

}  // namespace

std::tuple<Tensor, Tensor, Tensor> block(int64_t version, const Tensor &x_, const Tensor &shift_, const Tensor &state_,
                                         const std::vector<Tensor> &params, int64_t H, double eps, bool sync) {
    const Kind &k = kind_of(version);
    TORCH_CHECK_VALUE(params.size() == k.params, "wrong number of parameters");
    TORCH_CHECK_VALUE(x_.dim() == 3 && x_.size(1) > 0, "x must be [B,T,C] with T > 0");
    const int64_t B = x_.size(0), C = x_.size(2);
    TORCH_CHECK_VALUE(shift_.dim() == 2 && shift_.size(0) == B && shift_.size(1) == C, "the shift state must be [B,C]");
    // (nothing is launched before the state is known to fit: the kernels read it, and write its successor, by B and H)
    if (version == 4) {
        const int64_t A = params[P4_DECAY].numel();
        TORCH_CHECK_VALUE(state_.dim() == 3 && state_.size(0) == B && state_.size(1) == A && state_.size(2) == 3,
                          "the wkv state must be [", B, ",", A, ",3], got ", state_.sizes());
    } else {
        TORCH_CHECK_VALUE(state_.numel() == B * H * HEAD * HEAD, "the wkv state must be [", B, ",", H, ",64,64], got ", state_.sizes());
    }
    k.check(params, C, H);
    require_cuda({&x_, &shift_, &state_});
    for (const Tensor &p : params) require_cuda({&x_, &p});
    const Tensor x = x_.to(BF16).contiguous(), shift = shift_.to(BF16).contiguous();
    Tensor state = state_.to(at::kFloat).contiguous();
    if (version != 4 && state.sizes() != at::IntArrayRef({B, H, HEAD, HEAD})) state = state.view({B, H, HEAD, HEAD});
    bool grad = wants_grad({&x, &shift, &state});
    if (!grad && at::GradMode::is_enabled())
        for (const Tensor &p : params) grad |= p.requires_grad();
    if (grad) {
        variable_list in = {x, shift, state};
        in.insert(in.end(), params.begin(), params.end());
        auto node = make_node<BlockBackward>(in);
        node->version = version;
        node->meta = Meta{H, eps, sync};
        Out o;
        {
            at::AutoDispatchBelowADInplaceOrView below;
            c10::cuda::OptionalCUDAGuard guard(x.device());
            variable_list kept;
            o = k.forward(x, shift, state, params, node->meta, &kept);
            node->saved.reserve(in.size() + kept.size());
            for (const Tensor &t : in) node->keep({t});
            for (const Tensor &t : kept) node->keep({t});
        }
        torch::autograd::set_history(o.out, node);
        torch::autograd::set_history(o.shift, node);
        torch::autograd::set_history(o.state, node);
        return {o.out, o.shift, o.state};
    }
    at::AutoDispatchBelowADInplaceOrView below;
    c10::cuda::OptionalCUDAGuard guard(x.device());
    const Out o = k.forward(x, shift, state, params, Meta{H, eps, sync}, nullptr);
    return {o.out, o.shift, o.state};
}

}  // namespace wkv_native

void bind_blocks(py::module_ &m) { m.def("block", &wkv_native::block); }
