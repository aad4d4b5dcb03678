/* Entry points of libwkv_b200.so that only this package's own PyTorch binding calls: the public
 * ABI of wkv_b200.h with what a binding needs on top of it.  Not installed, not stable. */
#ifndef WKV_INTERNAL_H
#define WKV_INTERNAL_H

#include "../../include/wkv_b200.h"

#ifdef __cplusplus
extern "C" {
#endif

/* kernels this process has launched through the library */
unsigned long long wkvx_launch_count(void);

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

/* wkv_lnx_gate_* with parameters (and their gradients) in their own element type, and with silu != 0 the gate
 * silu(g): g is then the pre-activation and gg its gradient. */
int wkvx_lnx_gate_forward(int tokens, int H, const void *y, const void *g, const void *gamma, const void *beta, int param_dtype,
                          float eps, int silu, void *out, void *stream);
int wkvx_lnx_gate_backward(int tokens, int H, const void *y, const void *g, const void *gamma, const void *beta, int param_dtype,
                           float eps, int silu, const void *gout, void *gy, void *gg, void *ggamma, void *gbeta, void *workspace,
                           size_t workspace_bytes, void *stream);
/* wkv_ddlerp_* with one pointer per mix, in their own element type; one_minus: the parameters p_i stand for maa_i = 1 - p_i
 * (the gradients are w.r.t. p_i).  gx_add [B,T,C] and gshift_add [B,C] (or NULL) are added to gx and gshift_out. */
int wkvx_ddlerp_forward(int B, int T, int C, int nmix, const void *x, const void *shift, const void *const *maa, int maa_dtype,
                        int one_minus, const void *m, void *out, void *stream);
int wkvx_ddlerp_backward(int B, int T, int C, int nmix, const void *x, const void *shift, const void *const *maa, int maa_dtype,
                         int one_minus, const void *m, const void *gout, const void *gshift_in, const void *gx_add,
                         const void *gshift_add, void *gx, void *gm, void *gshift_out, void *const *gmaa, void *workspace,
                         size_t workspace_bytes, void *stream);

/* One token of a time-mix block for M rows (1 .. wkvx_decode_max_rows()), forward only (decode.cu).  bf16 tensors;
 * state fp32 [M,H,64,64] (key, value); C = H*64; scratch sizes beside the fields. */
int wkvx_decode_max_rows(void);
typedef struct wkvx_decode6 {
    int M, H, rank, decay_rank;             /* rank: 32 */
    const void *x, *shift;                  /* [M,C] */
    const void *maa_x, *maa[5];             /* [C]; w, k, v, r, g */
    int maa_dtype;
    const void *w1, *w2;                    /* [C,5*rank], [5,rank,C] */
    const void *decay, *d1, *d2;            /* [C], [C,decay_rank], [decay_rank,C] */
    const void *u;                          /* [H,64] */
    const void *proj[5];                    /* [C,C]: r, k, v, g, output */
    const void *ln_w, *ln_b;
    int ln_dtype;
    float eps;
    const float *state_in;
    void *t1, *xs, *rkvg, *dd, *normed;     /* [M,5*rank], [5,M,C], [4,M,C], [M,decay_rank], [M,C] */
    void *out, *new_shift;                  /* [M,C] */
    float *state_out;
} wkvx_decode6_t;
int wkvx_decode6(const wkvx_decode6_t *a, void *stream);

typedef struct wkvx_decode5 {
    int M, H, C;                            /* C: width of x and out; the attention width is H*64 */
    const void *x, *shift;                  /* [M,C] */
    const void *mix[4];                     /* [C]; k, v, r, g: maa = 1 - mix */
    int mix_dtype;
    const void *decay;                      /* [H,64] time_decay */
    int decay_dtype;
    const void *u;                          /* [H,64] */
    const void *proj[5];                    /* r, k, v, g [H*64,C], output [C,H*64] */
    const void *ln_w, *ln_b;
    int ln_dtype;
    float eps;
    const float *state_in;
    void *rkvg, *normed;                    /* [4,M,H*64], [M,H*64] */
    void *out, *new_shift;
    float *state_out;
} wkvx_decode5_t;
int wkvx_decode5(const wkvx_decode5_t *a, void *stream);

#ifdef __cplusplus
}
#endif
#endif
