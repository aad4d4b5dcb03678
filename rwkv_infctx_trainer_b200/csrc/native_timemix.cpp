// PyTorch binding of the op's elementwise neighbours (see timemix_fused.cu) as autograd nodes.
#include "native_ops.h"

namespace wkv_native {
namespace {

const Tensor &bf16(const Tensor &t, const char *name) {
    TORCH_CHECK_TYPE(t.scalar_type() == at::kBFloat16, name, " must be bfloat16");
    return t;
}

// the rows of a [n, C] parameter matrix
std::array<void *, 5> rows_of(const Tensor &t) {
    std::array<void *, 5> p{};
    for (int64_t i = 0; i < t.size(0) && i < 5; i++) p[i] = (char *)t.data_ptr() + i * t.size(1) * t.element_size();
    return p;
}

struct LnxGate : torch::autograd::Function<LnxGate> {
    static Tensor forward(AutogradContext *ctx, const Tensor &y_, const Tensor &g_, const Tensor &weight, const Tensor &bias,
                          double eps, int64_t H) {
        c10::cuda::OptionalCUDAGuard guard(y_.device());
        const auto pt = weight.scalar_type() == bias.scalar_type() ? param_type(weight) : at::kFloat;
        const Tensor y = contig(y_), g = contig(g_), ga = as_param(weight, pt), be = as_param(bias, pt);
        Tensor out = fresh_like(y);
        const int tokens = (int)(y.numel() / (H * HEAD));
        check(wkvx_lnx_gate_forward(tokens, (int)H, ptr(y), ptr(g), ptr(ga), ptr(be), dtype_code(pt), (float)eps, 0, ptr(out), stream_of(y)),
              "wkv_lnx_gate_forward");
        ctx->save_for_backward({y, g, ga, be});
        ctx->saved_data["eps"] = eps;
        ctx->saved_data["H"] = H;
        ctx->saved_data["types"] = std::vector<int64_t>{(int64_t)weight.scalar_type(), (int64_t)bias.scalar_type()};
        ctx->saved_data["w_shape"] = weight.sizes().vec();
        ctx->saved_data["b_shape"] = bias.sizes().vec();
        return out;
    }
    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const variable_list st = ctx->get_saved_variables();
        const Tensor &y = st[0], &g = st[1], &ga = st[2], &be = st[3];
        const int H = (int)ctx->saved_data["H"].toInt(), C = H * (int)HEAD, tokens = (int)(y.numel() / C);
        c10::cuda::OptionalCUDAGuard guard(y.device());
        const Tensor gout = as_contig(grads[0], at::kBFloat16);
        Tensor gy = fresh_like(y), gg = fresh_like(g), gga = fresh({C}, ga.scalar_type(), ga), gbe = fresh({C}, be.scalar_type(), be);
        const size_t n = wkv_lnx_gate_backward_workspace(tokens, H);
        Tensor ws = bytes_like(y, n);
        check(wkvx_lnx_gate_backward(tokens, H, ptr(y), ptr(g), ptr(ga), ptr(be), dtype_code(ga.scalar_type()),
                                     (float)ctx->saved_data["eps"].toDouble(), 0, ptr(gout), ptr(gy), ptr(gg), ptr(gga), ptr(gbe), ptr(ws), n,
                                     stream_of(y)),
              "wkv_lnx_gate_backward");
        const auto types = ctx->saved_data["types"].toIntVector();
        return {gy, gg, gga.view(ctx->saved_data["w_shape"].toIntVector()).to((at::ScalarType)types[0]),
                gbe.view(ctx->saved_data["b_shape"].toIntVector()).to((at::ScalarType)types[1]), Tensor(), Tensor()};
    }
};

struct DDLerp : torch::autograd::Function<DDLerp> {
    static Tensor forward(AutogradContext *ctx, const Tensor &x_, const Tensor &shift_, const Tensor &maa, const OptTensor &m_) {
        c10::cuda::OptionalCUDAGuard guard(x_.device());
        const Tensor x = contig(x_), sh = contig(shift_), m = m_.has_value() ? contig(*m_) : Tensor(), ma = as_param(maa, param_type(maa));
        const int B = (int)x.size(0), T = (int)x.size(1), C = (int)x.size(2), n = (int)ma.size(0);
        Tensor out = fresh({n, B, T, C}, x.scalar_type(), x);
        const auto p = rows_of(ma);
        check(wkvx_ddlerp_forward(B, T, C, n, ptr(x), ptr(sh), p.data(), dtype_code(ma.scalar_type()), 0, ptr(m), ptr(out), stream_of(x)),
              "wkv_ddlerp_forward");
        ctx->save_for_backward({x, sh, ma, m});
        ctx->saved_data["type"] = (int64_t)maa.scalar_type();
        return out;
    }
    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const variable_list st = ctx->get_saved_variables();
        const Tensor &x = st[0], &sh = st[1], &ma = st[2], &m = st[3];
        const int B = (int)x.size(0), T = (int)x.size(1), C = (int)x.size(2), n = (int)ma.size(0);
        c10::cuda::OptionalCUDAGuard guard(x.device());
        const Tensor gout = as_contig(grads[0], at::kBFloat16);
        Tensor gx = fresh_like(x), gm = m.defined() ? fresh_like(m) : Tensor(), gsh = fresh_like(sh),
               gma = fresh({n, C}, ma.scalar_type(), ma);
        const size_t nb = wkv_ddlerp_backward_workspace(B, T, C, n);
        Tensor ws = bytes_like(x, nb);
        const auto p = rows_of(ma), gp = rows_of(gma);
        check(wkvx_ddlerp_backward(B, T, C, n, ptr(x), ptr(sh), p.data(), dtype_code(ma.scalar_type()), 0, ptr(m), ptr(gout), nullptr, nullptr,
                                   nullptr, ptr(gx), ptr(gm), ptr(gsh), gp.data(), ptr(ws), nb, stream_of(x)),
              "wkv_ddlerp_backward");
        return {gx, gsh, gma.to((at::ScalarType)ctx->saved_data["type"].toInt()), gm};
    }
};

}  // namespace

Tensor lnx_gate(const Tensor &y, const Tensor &g, const Tensor &weight, const Tensor &bias, double eps, int64_t H) {
    require_cuda({&y, &g, &weight, &bias});
    const int64_t C = y.size(-1);
    TORCH_CHECK_VALUE(C == H * HEAD && g.sizes() == y.sizes() && weight.numel() == C && bias.numel() == C,
                      "y, g must be [..., n_head*64]; weight, bias [n_head*64]");
    return LnxGate::apply(bf16(y, "y"), bf16(g, "g"), weight, bias, eps, H);
}

Tensor ddlerp(const Tensor &x, const Tensor &shift, const Tensor &maa, const OptTensor &m_) {
    const Tensor m = m_.has_value() ? *m_ : Tensor();
    require_cuda({&x, &shift, &maa, &m});
    TORCH_CHECK_VALUE(x.dim() == 3 && maa.dim() == 2 && shift.dim() == 2, "x [B,T,C], shift [B,C], maa [n,C], m [n,B,T,C]");
    const int64_t B = x.size(0), T = x.size(1), C = x.size(2), n = maa.size(0);
    TORCH_CHECK_VALUE(maa.size(1) == C && shift.size(0) == B && shift.size(1) == C &&
                          (!m.defined() || (m.dim() == 4 && m.size(0) == n && m.size(1) == B && m.size(2) == T && m.size(3) == C)),
                      "x [B,T,C], shift [B,C], maa [n,C], m [n,B,T,C]");
    bf16(x, "x"); bf16(shift, "shift");
    if (m.defined()) bf16(m, "m");
    return DDLerp::apply(x, shift, maa, m_);
}

}  // namespace wkv_native

void bind_timemix(py::module_ &m) {
    m.def("lnx_gate", &wkv_native::lnx_gate);
    m.def("ddlerp", &wkv_native::ddlerp);
}
