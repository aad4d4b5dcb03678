/* Entry points of libwkv_b200.so that only this package's own PyTorch binding calls: the public
 * ABI of wkv_b200.h with what a binding needs on top of it.  Not installed, not stable. */
#ifndef WKV_INTERNAL_H
#define WKV_INTERNAL_H

#include "../../include/wkv_b200.h"

#ifdef __cplusplus
extern "C" {
#endif

/* wkv5/6_forward and _backward (per_token_w: 0 = v5, 1 = v6) with the status word at `status`
 * instead of the start of the workspace.  It may be mapped host memory; it is only ever written
 * when a device-side wait runs out and is not cleared by the call, so that a binding keeps one
 * word per device and looks at it without synchronising. */
int wkv56x_forward(const wkv_args_t *a, int per_token_w, int *status, void *stream);

/* The parameter gradients come summed over the batch, in a fixed order, in the element type of the
 * parameter (gu_sum [H,N]; v5: gw_sum [H,N]); a->gu (and v5's a->gw) are the per-batch partials of
 * the public call and may be NULL here. */
size_t wkv56x_backward_workspace(const wkv_args_t *a, int per_token_w);
int wkv56x_backward(const wkv_args_t *a, int per_token_w, int *status, void *gu_sum, int gu_dtype,
                    void *gw_sum, int gw_dtype, void *stream);

/* wkv4_forward_ckpt / wkv4_backward_ckpt from the time_decay parameter itself (any element type), without a
 * forward workspace, and with the parameter gradients summed over the batch in the parameters' types
 * (gw_sum [C] in decay_dtype, gu_sum [C] in gu_dtype).  state_ckpt: wkv4_state_ckpt_bytes() bytes or NULL. */
int wkv4x_forward(int B, int T, int C, int dtype, const void *time_decay, int decay_dtype, const void *u, const void *k,
                  const void *v, const float *state_in, void *y, float *state_out, void *state_ckpt, void *stream);
size_t wkv4x_backward_workspace(int B, int T, int C, int has_ckpt);
int wkv4x_backward(int B, int T, int C, int dtype, const void *time_decay, int decay_dtype, const void *u, const void *k,
                   const void *v, const float *state_in, const void *gy, const float *gstate_out, void *gw_sum, void *gu_sum,
                   int gu_dtype, void *gk, void *gv, float *gstate_in, void *workspace, const void *state_ckpt, void *stream);

#ifdef __cplusplus
}
#endif
#endif
