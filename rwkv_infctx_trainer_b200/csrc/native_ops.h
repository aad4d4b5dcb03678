// The v4/v5/v6 op calls of native_ops.cpp for the rest of the binding: no autograd, one call of the C ABI each.
#pragma once
#include "native_common.h"

namespace wkv_native {

struct Fwd {
    Tensor y, state_out, ckpt;
};
// saved_mode: WKV_GROUP_STATES_*; with it `saved` is the buffer (see wkv_args_t.group_states)
Fwd wkv56_forward(bool v6, const Tensor &r, const Tensor &k, const Tensor &v, const Tensor &w, const Tensor &u,
                  const Tensor &state_in, int w_kind, int layout, int path, const Tensor &state_out, bool save_ckpt,
                  int time_groups, const Tensor &saved, int saved_mode, bool sync_check);

struct Bwd {
    Tensor gr, gk, gv, gw, gu, gstate_in;
};
// gw: v6 [B,T,C] in r's type.  gu [H,64] in u's type and v5's gw [H,64] in `w_type` are summed over the
// batch; with per_batch they are the C ABI's fp32 [B,C] partials instead.
Bwd wkv56_backward(bool v6, const Tensor &r, const Tensor &k, const Tensor &v, const Tensor &w, const Tensor &u,
                   const Tensor &state_in, const Tensor &gy, const Tensor &gstate_out, int w_kind, int layout, int path,
                   bool want_gstate, const Tensor &ckpt, int time_groups, bool per_batch, at::ScalarType u_type,
                   at::ScalarType w_type, bool sync_check);

struct Fwd4 {
    Tensor y, state_out, ckpt;
};
// w (time_decay) in any element type of the ABI; u, k, v of one type; state fp32; all contiguous
Fwd4 wkv4_forward(const Tensor &w, const Tensor &u, const Tensor &k, const Tensor &v, const Tensor &state, bool save);
struct Bwd4 {
    Tensor gw, gu, gk, gv, gstate;
};
// gw in w's type, gu in `u_type`, both summed over the batch
Bwd4 wkv4_backward(const Tensor &w, const Tensor &u, const Tensor &k, const Tensor &v, const Tensor &state, const Tensor &ckpt,
                   const Tensor &gy, const Tensor &gstate_out, at::ScalarType u_type, bool want_gstate);

// the element type the ABI takes a parameter of this type in, and gives its gradient in (double: float)
inline at::ScalarType abi_type(at::ScalarType t) { return t == at::kBFloat16 || t == at::kHalf ? t : at::kFloat; }
inline at::ScalarType param_type(const Tensor &t) { return abi_type(t.scalar_type()); }

}  // namespace wkv_native
