// C-ABI entry points for v5/v6: argument validation and dispatch between the
// token-serial kernels and the chunked tensor-core kernels.
#include "wkv56_chunked.cuh"
#include "wkv_common.cuh"

#include "wkv_internal.h"

namespace wkv {
namespace {

// One CTA per (head, parameter): GROUPS groups of 16 threads (four channels each) take every GROUPS-th of the
// B*n rows, the groups meet in shared memory in a fixed order.  Latency-bound (a few hundred KB from
// L2): the width is there to have all loads of a few thousand tokens in flight at once (4 rows of 64 chunks x 64 heads:
// 7.5 us with 16 groups of one channel a thread and a division per row, 4.8 with this).
template <int GROUPS>
__global__ void __launch_bounds__(16 * GROUPS)
k_fold_heads(const float *__restrict__ gu_part, const float *__restrict__ gw_part, void *gu, int gu_dtype, void *gw,
             int gw_dtype, int B, int H, int n) {
    pdl_wait();
    pdl_trigger();
    __shared__ __align__(16) float red[GROUPS][64];
    __shared__ float red2[16][64];
    const int h = blockIdx.x, q = threadIdx.x & 15, g = threadIdx.x >> 4;
    const float *part = (blockIdx.y ? gw_part : gu_part) + (size_t)h * n * 64 + 4 * q;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    int b = g / n, j = g - b * n;
    const int step_b = GROUPS / n, step_j = GROUPS - step_b * n;
#pragma unroll 4
    for (int i = g; i < B * n; i += GROUPS) {
        const float4 v = *reinterpret_cast<const float4 *>(part + ((size_t)b * H * n + j) * 64);
        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
        b += step_b;
        j += step_j;
        if (j >= n) { j -= n; b++; }
    }
    *reinterpret_cast<float4 *>(&red[g][4 * q]) = acc;
    __syncthreads();
    const int k = threadIdx.x & 63, p = threadIdx.x >> 6;
    if (GROUPS > 16) {
        red2[p][k] = (red[4 * p][k] + red[4 * p + 1][k]) + (red[4 * p + 2][k] + red[4 * p + 3][k]);
        __syncthreads();
    }
    if (p == 0) {
        const float(*r)[64] = GROUPS > 16 ? red2 : red;
        float t = r[0][k];
#pragma unroll
        for (int i = 1; i < 16; i++) t += r[i][k];
        if (blockIdx.y) store_as(gw, gw_dtype, h * 64 + k, t);
        else store_as(gu, gu_dtype, h * 64 + k, t);
    }
}

// Up to a row for each of 16 groups: those alone, which start sooner and meet in one step (2, 8 and 16 rows: 2.95 us, with 64
// groups 3.26; 24 and 32 rows: 3.6 and 3.8, with 64 groups 3.5 and 3.6).
constexpr int FOLD_FEW_ROWS = 16;

}  // namespace

int fold_param_grads(const float *gu_part, const float *gw_part, int B, int H, int n, const CallOpts &opt, cudaStream_t s) {
    const bool few = (size_t)B * n <= FOLD_FEW_ROWS;
    return launch_chained(few ? k_fold_heads<16> : k_fold_heads<64>, dim3(H, gw_part ? 2 : 1), dim3(few ? 256 : 1024), 0, s, gu_part,
                          gw_part, opt.gu_sum, opt.gu_dtype, opt.gw_sum, opt.gw_dtype, B, H, n);
}

}  // namespace wkv

using namespace wkv;

namespace {

int check_common(const wkv_args_t *a, bool backward, bool per_token_w) {
    if (!a) return WKV_ERR_NULL;
    if (a->B < 0 || a->T < 0 || a->H < 0) return WKV_ERR_SHAPE;
    if (a->N != HEAD) return WKV_ERR_SHAPE;
    if (a->dtype != WKV_F32 && a->dtype != WKV_BF16 && a->dtype != WKV_F16) return WKV_ERR_DTYPE;
    if (a->w_kind != WKV_W_RAW && a->w_kind != WKV_W_NEGEXP) return WKV_ERR_DTYPE;
    if (a->state_layout != WKV_STATE_KV && a->state_layout != WKV_STATE_VK) return WKV_ERR_DTYPE;
    if (a->path != WKV_PATH_AUTO && a->path != WKV_PATH_SCALAR && a->path != WKV_PATH_CHUNKED)
        return WKV_ERR_DTYPE;
    if (a->time_groups < 0) return WKV_ERR_SHAPE;
    if (a->group_states_mode < WKV_GROUP_STATES_NONE || a->group_states_mode > WKV_GROUP_STATES_USE) return WKV_ERR_DTYPE;
    if (a->group_states && !aligned16(a->group_states)) return WKV_ERR_ALIGN;
    if (a->B == 0 || a->H == 0) return WKV_OK;
    if (!a->u) return WKV_ERR_NULL;
    if (!per_token_w && !a->w) return WKV_ERR_NULL;
    if (a->T > 0) {
        if (!a->r || !a->k || !a->v) return WKV_ERR_NULL;
        if (per_token_w && !a->w) return WKV_ERR_NULL;
        if (!backward && !a->y) return WKV_ERR_NULL;
        if (backward && (!a->gy || !a->gr || !a->gk || !a->gv)) return WKV_ERR_NULL;
        if (backward && per_token_w && !a->gw) return WKV_ERR_NULL;
    }
    if (backward && (!a->gu || (!per_token_w && !a->gw))) return WKV_ERR_NULL;
    const void *ptrs[] = {a->r, a->k, a->v, a->y, a->gy, a->gr, a->gk, a->gv, a->state_in,
                          a->state_out, a->gstate_out, a->gstate_in, a->workspace, a->state_ckpt};
    for (const void *p : ptrs)
        if (p && !aligned16(p)) return WKV_ERR_ALIGN;
    if (per_token_w && a->w && !aligned16(a->w)) return WKV_ERR_ALIGN;
    if (per_token_w && a->gw && !aligned16(a->gw)) return WKV_ERR_ALIGN;
    return WKV_OK;
}

bool use_chunked(const wkv_args_t *a, bool per_token_w, int *err) {
    *err = WKV_OK;
    if (a->path == WKV_PATH_SCALAR) return false;
    const bool ok = chunked_supported(a, per_token_w);
    if (a->path == WKV_PATH_CHUNKED && !ok) *err = WKV_ERR_UNSUPPORTED;
    return ok;
}

// (bf16, us, chunked against serial: 8 rows of 64 heads 35.6 / 15.5 at T = 32 and 36.9 / 28 at 64; one row of 8 heads 14 / 4.5
// and 14 / 7.4; 4 rows of 16 heads 14.4 / 6.6 and 14.4 / 16)
constexpr int SERIAL_MAX_T = 48;

size_t fwd_ws(const wkv_args_t *a, bool pt) {
    if (!a || a->B <= 0 || a->H <= 0 || a->T <= 0 || a->N != HEAD) return 0;
    int err;
    return use_chunked(a, pt, &err) ? chunked_forward_workspace(a, pt) : 0;
}

size_t bwd_ws(const wkv_args_t *a, bool pt) {
    if (!a || a->B <= 0 || a->H <= 0 || a->T <= 0 || a->N != HEAD) return 0;
    int err;
    return use_chunked(a, pt, &err) ? chunked_backward_workspace(a, pt) : scalar_backward_workspace(a);
}

int forward(const wkv_args_t *a, bool pt, void *stream, const CallOpts &opt = CallOpts()) {
    int err = check_common(a, false, pt);
    if (err != WKV_OK) return err;
    if (a->B == 0 || a->H == 0) return WKV_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const bool ch = use_chunked(a, pt, &err);
    if (err != WKV_OK) return err;
    const size_t need = fwd_ws(a, pt);
    if (need && (!a->workspace || a->workspace_bytes < need)) return WKV_ERR_WORKSPACE;
    if (ch && a->state_ckpt && a->state_ckpt_bytes < wkv56_state_ckpt_bytes(a, pt)) return WKV_ERR_WORKSPACE;
    if (a->group_states && a->group_states_mode != WKV_GROUP_STATES_NONE) {
        if (!ch) return WKV_ERR_UNSUPPORTED;
        if (a->group_states_bytes < wkv56_group_states_bytes(a)) return WKV_ERR_WORKSPACE;
    }
    // a call of a few tokens that leaves nothing for a backward pass (decode): the chunked kernel would pad
    // it to 64 tokens; the serial one reads and writes the state and little else
    if (ch && a->T <= SERIAL_MAX_T && a->path == WKV_PATH_AUTO && !a->state_ckpt && !a->group_states)
        return scalar_forward(a, pt, true, s);
    return ch ? chunked_forward(a, pt, opt, s) : scalar_forward(a, pt, false, s);
}

int backward(const wkv_args_t *a, bool pt, void *stream, const CallOpts &opt = CallOpts()) {
    int err = check_common(a, true, pt);
    if (err != WKV_OK) return err;
    if (a->B == 0 || a->H == 0) return WKV_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const bool ch = use_chunked(a, pt, &err);
    if (err != WKV_OK) return err;
    const size_t need = bwd_ws(a, pt);
    if (need && (!a->workspace || a->workspace_bytes < need)) return WKV_ERR_WORKSPACE;
    if (ch && a->state_ckpt && a->state_ckpt_bytes < wkv56_state_ckpt_bytes(a, pt)) return WKV_ERR_WORKSPACE;
    if (ch) return chunked_backward(a, pt, opt, s);
    err = scalar_backward(a, pt, s);
    if (err != WKV_OK || !opt.gu_sum) return err;
    return fold_param_grads(a->gu, pt ? nullptr : (const float *)a->gw, a->B, a->H, 1, opt, s);
}

}  // namespace

extern "C" {

const char *wkv_error_string(int code) {
    switch (code) {
        case WKV_OK: return "ok";
        case WKV_ERR_NULL: return "a required pointer is NULL";
        case WKV_ERR_SHAPE: return "bad shape (negative size or head size other than 64)";
        case WKV_ERR_DTYPE: return "unknown element type, decay encoding, state layout or path";
        case WKV_ERR_ALIGN: return "a tensor pointer is not 16-byte aligned";
        case WKV_ERR_WORKSPACE: return "workspace missing or too small";
        case WKV_ERR_LAUNCH: return "CUDA launch failed";
        case WKV_ERR_UNSUPPORTED: return "the chunked tensor-core path does not take these arguments";
        case WKV_ERR_TOO_LARGE: return "needs more scratch than the library's built-in array holds";
    }
    return "unknown error code";
}

int wkv56_uses_chunked(const wkv_args_t *a, int per_token_w);

unsigned long long wkvx_launch_count(void) { return launch_count.load(std::memory_order_relaxed); }

const char *wkv_version(void) { return "wkv_b200 2 sm_100a"; }

size_t wkv56_group_states_bytes(const wkv_args_t *a) {
    if (!a || a->B <= 0 || a->H <= 0 || a->T <= 0 || a->N != HEAD || a->dtype != WKV_BF16) return 0;
    return chunked_group_states_bytes(a);
}

size_t wkv56_state_ckpt_bytes(const wkv_args_t *a, int per_token_w) {
    if (!wkv56_uses_chunked(a, per_token_w)) return 0;
    return chunked::ckpt_layout(a->B, a->T, a->H).total;
}

int wkv56_uses_chunked(const wkv_args_t *a, int per_token_w) {
    if (!a || a->B <= 0 || a->H <= 0 || a->T <= 0 || a->N != HEAD) return 0;
    int err;
    return use_chunked(a, per_token_w != 0, &err) ? 1 : 0;
}

int wkv56x_forward(const wkv_args_t *a, int per_token_w, int *status, void *stream) {
    CallOpts opt;
    opt.status = status;
    return forward(a, per_token_w != 0, stream, opt);
}

// the per-batch partials of the public call go behind the workspace it asks for
size_t wkv56x_backward_workspace(const wkv_args_t *a, int per_token_w) {
    if (!a || a->B <= 0 || a->H <= 0 || a->N != HEAD) return 0;
    return ((bwd_ws(a, per_token_w != 0) + 255) & ~(size_t)255) + 2 * (size_t)a->B * a->H * HEAD * sizeof(float);
}

int wkv56x_backward(const wkv_args_t *a0, int per_token_w, int *status, void *gu_sum, int gu_dtype, void *gw_sum,
                    int gw_dtype, void *stream) {
    if (!a0 || !gu_sum || (!per_token_w && !gw_sum)) return WKV_ERR_NULL;
    const size_t need = wkv56x_backward_workspace(a0, per_token_w);
    if (need && (!a0->workspace || a0->workspace_bytes < need)) return WKV_ERR_WORKSPACE;
    if (need == 0) return WKV_OK;
    wkv_args_t a = *a0;
    float *partials = (float *)((char *)a.workspace + need) - 2 * (size_t)a.B * a.H * HEAD;
    a.gu = partials;
    if (!per_token_w) a.gw = partials + (size_t)a.B * a.H * HEAD;
    CallOpts opt;
    opt.status = status;
    opt.gu_sum = gu_sum; opt.gu_dtype = gu_dtype;
    opt.gw_sum = gw_sum; opt.gw_dtype = gw_dtype;
    return backward(&a, per_token_w != 0, stream, opt);
}

int wkv_selftest_wait_timeout(int *status_word, unsigned limit, void *stream) {
    if (!status_word) return WKV_ERR_NULL;
    return selftest_wait(status_word, limit, (cudaStream_t)stream);
}

int wkv56_selftest_abort(const wkv_args_t *a, int per_token_w, int backward_call, int kernel, int skip_chunk,
                         unsigned limit, void *stream) {
    if (limit == 0 || limit > 100000u || kernel < 0 || kernel > 2 || skip_chunk < 0) return WKV_ERR_SHAPE;
    if (!wkv56_uses_chunked(a, per_token_w)) return WKV_ERR_UNSUPPORTED;
    CallOpts opt;
    opt.wait_limit = limit;
    opt.kernel = kernel;
    opt.skip_load = skip_chunk;
    return backward_call ? backward(a, per_token_w != 0, stream, opt) : forward(a, per_token_w != 0, stream, opt);
}

size_t wkv5_forward_workspace(const wkv_args_t *a) { return fwd_ws(a, false); }
size_t wkv5_backward_workspace(const wkv_args_t *a) { return bwd_ws(a, false); }
int wkv5_forward(const wkv_args_t *a, void *stream) { return forward(a, false, stream); }
int wkv5_backward(const wkv_args_t *a, void *stream) { return backward(a, false, stream); }

size_t wkv6_forward_workspace(const wkv_args_t *a) { return fwd_ws(a, true); }
size_t wkv6_backward_workspace(const wkv_args_t *a) { return bwd_ws(a, true); }
int wkv6_forward(const wkv_args_t *a, void *stream) { return forward(a, true, stream); }
int wkv6_backward(const wkv_args_t *a, void *stream) { return backward(a, true, stream); }

}  // extern "C"
