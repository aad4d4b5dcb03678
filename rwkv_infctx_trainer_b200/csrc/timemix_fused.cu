// Elementwise neighbours of the WKV op in the v5/v6 time-mix block, fused so that every
// [B,T,C] tensor crosses HBM once per pass:
//
//   lnx_gate   out = GroupNorm_heads(y) * g      (RWKV-v6/src/module/TimeMix.py:296-298,
//              RWKV-v5/src/module/TimeMix.py:318-320: x = ln_x(x.view(-1,C)).view(B,T,C); x = x * g)
//              GroupNorm with one group per head: per token and head, the 64 channels are
//              normalised (biased variance, eps), then scaled and shifted per channel.
//   ddlerp     the five data-dependent token-shift mixes of v6
//              (RWKV-v6/src/module/TimeMix.py:262-273):  x_i = x + (x_prev - x) * (maa_i + m_i)
//
// All are HBM-bound: a thread owns 8 consecutive channels (one 16-byte access per tensor), the 8
// lanes that share a head exchange their sums by shuffles, accumulation is fp32, parameter
// gradients are reduced in a fixed order (per-CTA partials, then one fold): no atomics.
// Parameters come in their own element type and from their own tensors (a block's mixes are
// separate parameters), and their gradients go back the same way.
#include <initializer_list>
#include <type_traits>

#include "wkv_common.cuh"
#include "wkv_internal.h"

namespace wkv {
namespace {

constexpr int TPB = 256;

// sum over the 8 lanes that hold one head's 64 channels
__device__ __forceinline__ float head_sum(float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    return v;
}
// 8 channels of a parameter of element type `dtype`
__device__ __forceinline__ void load8(const void *p, int dtype, size_t at, float *f) {
    if (dtype == WKV_BF16) {
        unpack8(__ldg(reinterpret_cast<const uint4 *>((const __nv_bfloat16 *)p + at)), f);
    } else if (dtype == WKV_F32) {
        const float4 *q = reinterpret_cast<const float4 *>((const float *)p + at);
        const float4 a = __ldg(q), b = __ldg(q + 1);
        f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
    } else {
        const __half2 *q = reinterpret_cast<const __half2 *>((const __half *)p + at);
#pragma unroll
        for (int i = 0; i < 4; i++) { const float2 v = __half22float2(q[i]); f[2 * i] = v.x; f[2 * i + 1] = v.y; }
    }
}

// Work split shared by the kernels: the C channels are cut into column blocks of 256 (a warp's
// 32 lanes x 8 channels = 4 heads); blockIdx.x = column block + ncb * token slot; the 8 warps of
// a CTA take tokens slot*8 + warp, slot*8 + warp + stride, ...  A thread therefore always owns the
// same 8 channels, which keeps its parameters and its parameter-gradient sums in registers.
struct Split {
    int ncb, nslot;
};
constexpr int LNX_FWD_CTAS = 5, LNX_BWD_CTAS = 3;

// SILU: the gate is silu(g), rounded to bf16 as the tensor it stands for would be
template <bool SILU>
__global__ void __launch_bounds__(TPB, LNX_FWD_CTAS)
k_lnx_gate_fwd(int tokens, int C, Split sp, const uint4 *__restrict__ y, const uint4 *__restrict__ g,
               const void *__restrict__ gamma, const void *__restrict__ beta, int pdtype, float eps, uint4 *__restrict__ out) {
    pdl_wait();
    pdl_trigger();
    const int cb = blockIdx.x % sp.ncb, slot = blockIdx.x / sp.ncb, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c0 = cb * 256 + lane * 8;
    // (lanes past the last channel stay in the loop with zeros: the shuffles below name all 32 lanes)
    const bool live = c0 < C;
    float ga[8], be[8];
#pragma unroll
    for (int q = 0; q < 8; q++) { ga[q] = 0.f; be[q] = 0.f; }
    if (live) {
        load8(gamma, pdtype, c0, ga);
        load8(beta, pdtype, c0, be);
    }
    const int stride = sp.nslot * 8, row16 = C / 8;
    const uint4 zero4 = make_uint4(0u, 0u, 0u, 0u);
    uint4 raw[2] = {zero4, zero4};       // the next token's, on their way while this one is worked on
    auto fetch = [&](int t) {
        const size_t i = (size_t)t * row16 + (c0 >> 3);
        if (live && t < tokens) { raw[0] = y[i]; raw[1] = g[i]; }
    };
    fetch(slot * 8 + warp);
    for (int t = slot * 8 + warp; t < tokens; t += stride) {
        const size_t i = (size_t)t * row16 + (c0 >> 3);
        float yv[8], gv[8];
        unpack8(raw[0], yv);
        unpack8(raw[1], gv);
        fetch(t + stride);
        if (SILU) {
#pragma unroll
            for (int q = 0; q < 8; q++) gv[q] = bf16_round(gv[q] * sigmoidf(gv[q]));
        }
        float s = 0.f;
#pragma unroll
        for (int q = 0; q < 8; q++) s += yv[q];
        const float mean = head_sum(s) * (1.f / 64.f);
        float v = 0.f;
#pragma unroll
        for (int q = 0; q < 8; q++) { yv[q] -= mean; v += yv[q] * yv[q]; }
        const float rstd = rsqrtf(head_sum(v) * (1.f / 64.f) + eps);
        float o[8];
#pragma unroll
        for (int q = 0; q < 8; q++) o[q] = (yv[q] * rstd * ga[q] + be[q]) * gv[q];
        if (live) out[i] = pack8(o);
    }
}

// gy, gg and per-CTA partial sums of the gradients of gamma and beta ([nslot, 2, C])
template <bool SILU>
__global__ void __launch_bounds__(TPB, LNX_BWD_CTAS)
k_lnx_gate_bwd(int tokens, int C, Split sp, const uint4 *__restrict__ y, const uint4 *__restrict__ g,
               const void *__restrict__ gamma, const void *__restrict__ beta, int pdtype, float eps,
               const uint4 *__restrict__ gout, uint4 *__restrict__ gy, uint4 *__restrict__ gg,
               float *__restrict__ part) {
    pdl_wait();
    pdl_trigger();
    __shared__ __align__(16) float red[8][2][256];
    const int cb = blockIdx.x % sp.ncb, slot = blockIdx.x / sp.ncb, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c0 = cb * 256 + lane * 8;
    const bool live = c0 < C;
    float dga[8], dbe[8];
#pragma unroll
    for (int q = 0; q < 8; q++) { dga[q] = 0.f; dbe[q] = 0.f; }
    {
        // (every lane runs the loop, lanes past the last channel on zeros: the shuffles name all 32 lanes)
        // gamma and beta wait in shared memory, each warp's own copy: the registers go to the loads ahead
        float *gab = &red[warp][0][lane * 8], *beb = &red[warp][1][lane * 8];
        {
            float ga[8], be[8];
#pragma unroll
            for (int q = 0; q < 8; q++) { ga[q] = 0.f; be[q] = 0.f; }
            if (live) {
                load8(gamma, pdtype, c0, ga);
                load8(beta, pdtype, c0, be);
            }
#pragma unroll
            for (int q = 0; q < 8; q++) { gab[q] = ga[q]; beb[q] = be[q]; }
        }
        const int stride = sp.nslot * 8, row16 = C / 8;
        const uint4 zero4 = make_uint4(0u, 0u, 0u, 0u);
        uint4 raw[3] = {zero4, zero4, zero4};       // the next token's, on their way while this one is worked on
        auto fetch = [&](int t) {
            const size_t i = (size_t)t * row16 + (c0 >> 3);
            if (live && t < tokens) { raw[0] = y[i]; raw[1] = g[i]; raw[2] = gout[i]; }
        };
        fetch(slot * 8 + warp);
        for (int t = slot * 8 + warp; t < tokens; t += stride) {
            const size_t i = (size_t)t * row16 + (c0 >> 3);
            float yv[8], gv[8], go[8];
            unpack8(raw[0], yv);
            unpack8(raw[1], gv);
            unpack8(raw[2], go);
            fetch(t + stride);
            float dsilu[8];
            if (SILU) {
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const float sg = sigmoidf(gv[q]);
                    dsilu[q] = sg * (1.f + gv[q] * (1.f - sg));
                    gv[q] = bf16_round(gv[q] * sg);
                }
            }
            float s = 0.f;
#pragma unroll
            for (int q = 0; q < 8; q++) s += yv[q];
            const float mean = head_sum(s) * (1.f / 64.f);
            float v = 0.f;
#pragma unroll
            for (int q = 0; q < 8; q++) { yv[q] -= mean; v += yv[q] * yv[q]; }
            const float rstd = rsqrtf(head_sum(v) * (1.f / 64.f) + eps);
            float dg[8], dy[8], s1 = 0.f, s2 = 0.f, ga[8], be[8];
#pragma unroll
            for (int q = 0; q < 8; q += 4) {
                const float4 p = *reinterpret_cast<const float4 *>(gab + q), r = *reinterpret_cast<const float4 *>(beb + q);
                ga[q] = p.x; ga[q + 1] = p.y; ga[q + 2] = p.z; ga[q + 3] = p.w;
                be[q] = r.x; be[q + 1] = r.y; be[q + 2] = r.z; be[q + 3] = r.w;
            }
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const float xh = yv[q] * rstd;               // normalised value
                const float dln = go[q] * gv[q];             // gradient at the GroupNorm output
                dg[q] = go[q] * (xh * ga[q] + be[q]);
                if (SILU) dg[q] *= dsilu[q];
                dga[q] += dln * xh;
                dbe[q] += dln;
                dy[q] = dln * ga[q];                         // gradient at the normalised value
                s1 += dy[q];
                s2 += dy[q] * xh;
                yv[q] = xh;
            }
            const float m1 = head_sum(s1) * (1.f / 64.f), m2 = head_sum(s2) * (1.f / 64.f);
#pragma unroll
            for (int q = 0; q < 8; q++) dy[q] = rstd * (dy[q] - m1 - yv[q] * m2);
            if (live) {
                gy[i] = pack8(dy);
                gg[i] = pack8(dg);
            }
        }
    }
    // the CTA's 8 warps hold partial sums for the same 256 channels: fold them in warp order
#pragma unroll
    for (int q = 0; q < 8; q++) { red[warp][0][lane * 8 + q] = dga[q]; red[warp][1][lane * 8 + q] = dbe[q]; }
    __syncthreads();
    const int c = cb * 256 + threadIdx.x;
    if (c < C) {
        float a = 0.f, b = 0.f;
#pragma unroll
        for (int w = 0; w < 8; w++) { a += red[w][0][threadIdx.x]; b += red[w][1][threadIdx.x]; }
        part[((size_t)slot * 2) * C + c] = a;
        part[((size_t)slot * 2 + 1) * C + c] = b;
    }
}

// Column sums of the per-CTA partials [rows, n*C] into n parameter gradients of C elements: 32 columns by 8 row groups
// per CTA, many loads in flight; `sign` -1 for parameters that enter as 1 - p.
struct GradPtrs {
    void *p[5];
};
__global__ void __launch_bounds__(TPB)
k_fold_cols(const float *__restrict__ part, int rows, int n, int C, GradPtrs out, int dtype, float sign) {
    pdl_wait();
    pdl_trigger();
    __shared__ float red[8][32];
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5, col = blockIdx.x * 32 + lane, cols = n * C;
    float a = 0.f;
    if (col < cols) {
#pragma unroll 8
        for (int r = g; r < rows; r += 8) a += part[(size_t)r * cols + col];
    }
    red[g][lane] = a;
    __syncthreads();
    if (g == 0 && col < cols) {
#pragma unroll
        for (int q = 1; q < 8; q++) a += red[q][lane];
        store_as(out.p[col / C], dtype, col % C, sign * a);
    }
}

// x_i = x + (x_prev - x) * (maa_i + m_i) for n mixes; x_prev of a row's first token is `shift` (the
// last token of the previous segment).  m: [n, tokens, C] (NULL: no data-dependent part).
struct MixPtrs {
    const void *p[5];       // maa_i, [C] each
    int dtype;
    int one_minus;          // the parameters are 1 - maa_i
    __device__ __forceinline__ void load(int n, int c, float *f) const {
        load8(p[n], dtype, c, f);
        if (one_minus) {
#pragma unroll
            for (int q = 0; q < 8; q++) f[q] = 1.f - f[q];
        }
    }
};
template <int NMIX>
__global__ void __launch_bounds__(TPB)
k_ddlerp_fwd(int B, int T, int C, const uint4 *__restrict__ x, const uint4 *__restrict__ shift, const MixPtrs maa,
             const uint4 *__restrict__ m, uint4 *__restrict__ out) {
    pdl_wait();
    pdl_trigger();
    const int row16 = C / 8;
    const size_t total = (size_t)B * T * row16, tokens = (size_t)B * T;
    for (size_t i = (size_t)blockIdx.x * TPB + threadIdx.x; i < total; i += (size_t)gridDim.x * TPB) {
        const size_t tok = i / row16;
        const int c8 = (int)(i - tok * row16), t = (int)(tok % T), b = (int)(tok / T);
        float xv[8], pv[8];
        unpack8(x[i], xv);
        unpack8(t > 0 ? x[i - row16] : shift[(size_t)b * row16 + c8], pv);
#pragma unroll
        for (int q = 0; q < 8; q++) pv[q] -= xv[q];
#pragma unroll
        for (int n = 0; n < NMIX; n++) {
            float a[8], mv[8], o[8];
            maa.load(n, c8 * 8, a);
            if (m) {
                unpack8(m[(size_t)n * tokens * row16 + i], mv);
#pragma unroll
                for (int q = 0; q < 8; q++) a[q] += mv[q];
            }
#pragma unroll
            for (int q = 0; q < 8; q++) o[q] = xv[q] + pv[q] * a[q];
            out[(size_t)n * tokens * row16 + i] = pack8(o);
        }
    }
}

// Backward of the mixes: with d = x_prev - x and a_i = maa_i + m_i,
//   gm_i = gout_i * d,   gmaa_i = sum over tokens of gm_i,
//   gx_t = sum_i gout_i,t (1 - a_i,t)  +  sum_i gout_i,t+1 a_i,t+1     (the second term: token t is
//   the predecessor of t+1; for a row's last token it comes from the next segment, `gshift_in`),
//   gshift_out = sum_i gout_i,0 a_i,0   (gradient w.r.t. `shift`).
// A warp walks `sub` consecutive tokens of 256 channels backward, so that the t+1 term is carried in registers; the 8
// warps of a CTA take 8*sub consecutive tokens of the same channels, hand that term on through shared memory (only the
// CTA's last warp forms its first one from the token after it) and pool their sums of gm for gmaa.  HBM-bound: the
// loads of K tokens go out before the first is used, and `sub` is chosen so that the grid is one wave, or as
// few as possible (ddlerp_sub).  4096 x 2560 tokens, 5 mixes, 17 tensors of 21 MB, of which 64-token CTAs
// in 2.2 waves took 116 us: 81 us; one mix, 4 tensors: 36 -> 21 us.
// gx_add, gshift_add: gradients of x and shift from elsewhere, added.
constexpr int MIX_CTAS = 2;       // per SM
template <int NMIX>
__global__ void __launch_bounds__(TPB, MIX_CTAS)
k_ddlerp_bwd(int B, int T, int C, int sub, const uint4 *__restrict__ x, const uint4 *__restrict__ shift, const MixPtrs maa,
             const uint4 *__restrict__ m, const uint4 *__restrict__ gout, const uint4 *__restrict__ gshift_in,
             const uint4 *__restrict__ gx_add, const uint4 *__restrict__ gshift_add, uint4 *__restrict__ gx,
             uint4 *__restrict__ gm, uint4 *__restrict__ gshift_out, float *__restrict__ part) {
    pdl_wait();
    pdl_trigger();
    constexpr int K = NMIX == 1 ? 4 : 1;
    __shared__ __align__(16) float red[8][256];
    __shared__ __align__(16) float last[8][256];          // gx of a warp's last token without the term from its successor
    __shared__ __align__(16) float mixes[NMIX][256];      // maa of the CTA's channels
    const int row16 = C / 8, ncb = (C + 255) / 256, npiece = (T + 8 * sub - 1) / (8 * sub);
    const int cb = blockIdx.x % ncb, rowp = blockIdx.x / ncb, b = rowp / npiece, pc = rowp - b * npiece;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c8 = cb * 32 + lane;
    const size_t tokens16 = (size_t)B * T * row16, base = (size_t)b * T * row16 + c8;
    const int t0 = pc * 8 * sub + warp * sub, t1 = min(T, t0 + sub);
    const bool act = c8 < row16 && t0 < T;
    for (int k = threadIdx.x; k < NMIX * 32; k += TPB) {
        const int n = k >> 5, l = k & 31;
        if (cb * 32 + l < row16) maa.load(n, (cb * 32 + l) * 8, &mixes[n][l * 8]);
    }
    __syncthreads();
    auto lds8 = [&](const float *row, float *a) {
        const float4 p = *reinterpret_cast<const float4 *>(row + lane * 8), q = *reinterpret_cast<const float4 *>(row + lane * 8 + 4);
        a[0] = p.x; a[1] = p.y; a[2] = p.z; a[3] = p.w; a[4] = q.x; a[5] = q.y; a[6] = q.z; a[7] = q.w;
    };
    auto sts8 = [&](float *row, const float *a) {
        *reinterpret_cast<float4 *>(row + lane * 8) = make_float4(a[0], a[1], a[2], a[3]);
        *reinterpret_cast<float4 *>(row + lane * 8 + 4) = make_float4(a[4], a[5], a[6], a[7]);
    };
    float acc[NMIX][8], carry[8];
#pragma unroll
    for (int q = 0; q < 8; q++) {
        carry[q] = 0.f;
#pragma unroll
        for (int n = 0; n < NMIX; n++) acc[n][q] = 0.f;
    }
    if (act) {
        uint4 xraw = x[base + (size_t)(t1 - 1) * row16];
        auto walk = [&](int t, auto count) {         // tokens t, t-1, ...
            constexpr int N = decltype(count)::value;
            uint4 graw[N][NMIX], mraw[N][NMIX], praw[N], araw[N];
#pragma unroll
            for (int k = 0; k < N; k++) {
                const size_t i = base + (size_t)(t - k) * row16;
#pragma unroll
                for (int n = 0; n < NMIX; n++) {
                    graw[k][n] = gout[n * tokens16 + i];
                    if (m) mraw[k][n] = m[n * tokens16 + i];
                }
                praw[k] = t - k > 0 ? x[i - row16] : shift[(size_t)b * row16 + c8];
                if (NMIX == 1 && gx_add) araw[k] = gx_add[i];
            }
#pragma unroll
            for (int k = 0; k < N; k++) {
                const size_t i = base + (size_t)(t - k) * row16;
                float xv[8], d[8], gxv[8], nxt[8];
                unpack8(xraw, xv);
                unpack8(praw[k], d);
                vsub<8>(d, d, xv);
                if (gx_add) {
                    unpack8(NMIX == 1 ? araw[k] : gx_add[i], gxv);
                    vadd<8>(gxv, gxv, carry);
                } else {
#pragma unroll
                    for (int q = 0; q < 8; q++) gxv[q] = carry[q];
                }
#pragma unroll
                for (int q = 0; q < 8; q++) nxt[q] = 0.f;
#pragma unroll
                for (int n = 0; n < NMIX; n++) {
                    float go[8], a[8], gmv[8];
                    unpack8(graw[k][n], go);
                    lds8(mixes[n], a);
                    if (m) {
                        float mv[8];
                        unpack8(mraw[k][n], mv);
                        vadd<8>(a, a, mv);
                    }
                    vmul<8>(gmv, go, d);
                    vadd<8>(acc[n], acc[n], gmv);
                    vmul<8>(a, a, go);
                    vadd<8>(nxt, nxt, a);
                    vsub<8>(a, go, a);
                    vadd<8>(gxv, gxv, a);
                    if (gm) gm[n * tokens16 + i] = pack8(gmv);
                }
                if (t - k == t1 - 1) sts8(last[warp], gxv);
                else gx[i] = pack8(gxv);
#pragma unroll
                for (int q = 0; q < 8; q++) carry[q] = nxt[q];
                xraw = praw[k];
            }
        };
        int t = t1 - 1;
        if (K > 1) {
#pragma unroll 1
            for (; t - K + 1 >= t0; t -= K) walk(t, std::integral_constant<int, K>());
        }
#pragma unroll 1
        for (; t >= t0; t--) walk(t, std::integral_constant<int, 1>());
        if (t0 == 0 && gshift_out) {
            float out[8], add[8];
            if (gshift_add) unpack8(gshift_add[(size_t)b * row16 + c8], add);
#pragma unroll
            for (int q = 0; q < 8; q++) out[q] = carry[q] + (gshift_add ? add[q] : 0.f);
            gshift_out[(size_t)b * row16 + c8] = pack8(out);
        }
    }
    // what the warp's first token sends back goes to the warp before; each finishes its last token
    sts8(red[warp], carry);
    __syncthreads();
    if (act) {
        float end[8];
        lds8(last[warp], end);
        if (t1 < T && warp < 7) {
            float g[8];
            lds8(red[warp + 1], g);
            vadd<8>(end, end, g);
        } else if (t1 < T) {
            const size_t j = base + (size_t)t1 * row16;
#pragma unroll
            for (int n = 0; n < NMIX; n++) {
                float go[8], a[8];
                unpack8(gout[n * tokens16 + j], go);
                lds8(mixes[n], a);
                if (m) {
                    float mv[8];
                    unpack8(m[n * tokens16 + j], mv);
                    vadd<8>(a, a, mv);
                }
                vfma<8>(end, go, a, end);
            }
        } else if (gshift_in) {
            float g[8];
            unpack8(gshift_in[(size_t)b * row16 + c8], g);
            vadd<8>(end, end, g);
        }
        gx[base + (size_t)(t1 - 1) * row16] = pack8(end);
    }
    // the CTA's sums of gm per mix: [B*npiece, NMIX, C], folded by k_fold_cols
#pragma unroll 1
    for (int n = 0; n < NMIX; n++) {
        __syncthreads();
#pragma unroll
        for (int k = 0; k < NMIX; k++)
            if (k == n) {
#pragma unroll
                for (int q = 0; q < 8; q++) red[warp][(lane * 8 + q) ^ (lane & 7)] = acc[k][q];
            }
        __syncthreads();
        const int c = cb * 256 + threadIdx.x, sw = (threadIdx.x) ^ ((threadIdx.x >> 3) & 7);
        if (c < C) {
            float a = 0.f;
#pragma unroll
            for (int w = 0; w < 8; w++) a += red[w][sw];
            part[((size_t)rowp * NMIX + n) * C + c] = a;
        }
    }
}

// ctas: as many per SM as are resident at once; the tokens come through a loop that loads ahead, and in backward every
// CTA leaves a row of partials to fold.  4096 x 2560 tokens: forward 11.0 -> 9.7 us, backward 37 + 10 ->
// 28 + 8 us.
Split make_split(int tokens, int C, int ctas) {
    Split sp;
    sp.ncb = (C + 255) / 256;
    const int want = device_sm_count() * ctas / sp.ncb;
    const int most = (tokens + 7) / 8;
    sp.nslot = want < most ? want : most;
    if (sp.nslot < 1) sp.nslot = 1;
    return sp;
}

// How k_ddlerp_bwd cuts a row: tokens per warp.  All CTAs of a wave walk side by side, so a grid a little over one
// wave costs two; of one to eight waves the cut with the fewest token steps (and two for a CTA's start and end).
int ddlerp_sub(int B, int T, int C) {
    const long long cols = (long long)B * ((C + 255) / 256), slots = (long long)device_sm_count() * MIX_CTAS;
    int best = 0;
    long long least = 0;
    for (int w = 1; w <= 8; w++) {
        long long pieces = w * slots / cols;
        if (pieces < 1) pieces = 1;
        long long sub = (T + 8 * pieces - 1) / (8 * pieces);
        if (sub < 2) sub = 2;
        const long long ctas = cols * ((T + 8 * sub - 1) / (8 * sub)), cost = (ctas + slots - 1) / slots * (sub + 2);
        if (best == 0 || cost < least) { best = (int)sub; least = cost; }
        if (sub == 2) break;
    }
    return best;
}
size_t ddlerp_rows(int B, int T, int C) {
    const int piece = 8 * ddlerp_sub(B, T, C);
    return (size_t)B * ((T + piece - 1) / piece);
}

int fold_cols(const float *part, size_t rows, int n, int C, void *const *out, int dtype, float sign, cudaStream_t s) {
    GradPtrs g = {};
    for (int i = 0; i < n; i++) g.p[i] = out[i];
    return launch_chained(k_fold_cols, dim3((n * C + 31) / 32), dim3(TPB), 0, s, part, (int)rows, n, C, g, dtype, sign);
}

template <int NMIX>
int ddlerp_bwd_launch(int B, int T, int C, const void *x, const void *shift, const MixPtrs &maa, const void *m, const void *gout,
                      const void *gshift_in, const void *gx_add, const void *gshift_add, void *gx, void *gm, void *gshift_out,
                      float *part, cudaStream_t s) {
    const dim3 grid((unsigned)(ddlerp_rows(B, T, C) * ((C + 255) / 256)));
    return launch_chained(k_ddlerp_bwd<NMIX>, grid, dim3(TPB), 0, s, B, T, C, ddlerp_sub(B, T, C), (const uint4 *)x, (const uint4 *)shift,
                          maa, (const uint4 *)m, (const uint4 *)gout, (const uint4 *)gshift_in, (const uint4 *)gx_add,
                          (const uint4 *)gshift_add, (uint4 *)gx, (uint4 *)gm, (uint4 *)gshift_out, part);
}
template <int NMIX>
int ddlerp_fwd_launch(int B, int T, int C, const void *x, const void *shift, const MixPtrs &maa, const void *m, void *out, cudaStream_t s) {
    const size_t total = (size_t)B * T * (C / 8);
    size_t blocks = (total + TPB - 1) / TPB;
    if (blocks > 148 * 16) blocks = 148 * 16;
    return launch_chained(k_ddlerp_fwd<NMIX>, dim3((unsigned)blocks), dim3(TPB), 0, s, B, T, C, (const uint4 *)x, (const uint4 *)shift, maa,
                          (const uint4 *)m, (uint4 *)out);
}

bool mixes_ok(int n) { return n == 1 || n == 3 || n == 4 || n == 5; }
MixPtrs mix_ptrs(int n, const void *const *maa, int dtype, int one_minus) {
    MixPtrs p = {};
    for (int i = 0; i < n; i++) p.p[i] = maa[i];
    p.dtype = dtype;
    p.one_minus = one_minus;
    return p;
}
}  // namespace
}  // namespace wkv

using namespace wkv;

extern "C" {

int wkvx_lnx_gate_forward(int tokens, int H, const void *y, const void *g, const void *gamma, const void *beta, int param_dtype,
                          float eps, int silu, void *out, void *stream) {
    if (tokens < 0 || H < 0) return WKV_ERR_SHAPE;
    if (tokens == 0 || H == 0) return WKV_OK;
    if (!y || !g || !gamma || !beta || !out) return WKV_ERR_NULL;
    if (!all_aligned({y, g, gamma, beta, out})) return WKV_ERR_ALIGN;
    const int C = H * HEAD;
    const Split sp = make_split(tokens, C, LNX_FWD_CTAS);
    return launch_chained(silu ? k_lnx_gate_fwd<true> : k_lnx_gate_fwd<false>, dim3(sp.ncb * sp.nslot), dim3(TPB), 0, (cudaStream_t)stream,
                          tokens, C, sp, (const uint4 *)y, (const uint4 *)g, gamma, beta, param_dtype, eps, (uint4 *)out);
}

int wkv_lnx_gate_forward(int tokens, int H, const void *y, const void *g, const float *gamma, const float *beta,
                         float eps, void *out, void *stream) {
    return wkvx_lnx_gate_forward(tokens, H, y, g, gamma, beta, WKV_F32, eps, 0, out, stream);
}

size_t wkv_lnx_gate_backward_workspace(int tokens, int H) {
    if (tokens <= 0 || H <= 0) return 0;
    return (size_t)make_split(tokens, H * HEAD, LNX_BWD_CTAS).nslot * 2 * H * HEAD * sizeof(float);
}

int wkvx_lnx_gate_backward(int tokens, int H, const void *y, const void *g, const void *gamma, const void *beta, int param_dtype,
                           float eps, int silu, const void *gout, void *gy, void *gg, void *ggamma, void *gbeta, void *workspace,
                           size_t workspace_bytes, void *stream) {
    if (tokens < 0 || H < 0) return WKV_ERR_SHAPE;
    if (H == 0) return WKV_OK;
    if (!ggamma || !gbeta) return WKV_ERR_NULL;
    const int C = H * HEAD;
    cudaStream_t s = (cudaStream_t)stream;
    if (tokens == 0) {
        const size_t n = (size_t)C * (param_dtype == WKV_F32 ? 4 : 2);
        if (cudaMemsetAsync(ggamma, 0, n, s) != cudaSuccess || cudaMemsetAsync(gbeta, 0, n, s) != cudaSuccess) return WKV_ERR_LAUNCH;
        return WKV_OK;
    }
    if (!y || !g || !gamma || !beta || !gout || !gy || !gg) return WKV_ERR_NULL;
    if (!all_aligned({y, g, gamma, beta, gout, gy, gg})) return WKV_ERR_ALIGN;
    if (!workspace || workspace_bytes < wkv_lnx_gate_backward_workspace(tokens, H)) return WKV_ERR_WORKSPACE;
    const Split sp = make_split(tokens, C, LNX_BWD_CTAS);
    if (launch_chained(silu ? k_lnx_gate_bwd<true> : k_lnx_gate_bwd<false>, dim3(sp.ncb * sp.nslot), dim3(TPB), 0, s, tokens, C, sp,
                       (const uint4 *)y, (const uint4 *)g, gamma, beta, param_dtype, eps, (const uint4 *)gout, (uint4 *)gy, (uint4 *)gg,
                       (float *)workspace) != WKV_OK)
        return WKV_ERR_LAUNCH;
    void *out[2] = {ggamma, gbeta};
    return fold_cols((const float *)workspace, sp.nslot, 2, C, out, param_dtype, 1.f, s);
}

int wkv_lnx_gate_backward(int tokens, int H, const void *y, const void *g, const float *gamma, const float *beta,
                          float eps, const void *gout, void *gy, void *gg, float *ggamma, float *gbeta,
                          void *workspace, size_t workspace_bytes, void *stream) {
    return wkvx_lnx_gate_backward(tokens, H, y, g, gamma, beta, WKV_F32, eps, 0, gout, gy, gg, ggamma, gbeta, workspace, workspace_bytes, stream);
}

int wkvx_ddlerp_forward(int B, int T, int C, int nmix, const void *x, const void *shift, const void *const *maa, int maa_dtype,
                        int one_minus, const void *m, void *out, void *stream) {
    if (B < 0 || T < 0 || C < 0 || C % 8 != 0) return WKV_ERR_SHAPE;
    if (!mixes_ok(nmix)) return WKV_ERR_UNSUPPORTED;
    if (B == 0 || T == 0 || C == 0) return WKV_OK;
    if (!x || !shift || !maa || !out) return WKV_ERR_NULL;
    for (int i = 0; i < nmix; i++)
        if (!maa[i]) return WKV_ERR_NULL;
        else if (!aligned16(maa[i])) return WKV_ERR_ALIGN;
    if (!all_aligned({x, shift, out, m})) return WKV_ERR_ALIGN;
    const MixPtrs p = mix_ptrs(nmix, maa, maa_dtype, one_minus);
    cudaStream_t s = (cudaStream_t)stream;
    switch (nmix) {
        case 5: return ddlerp_fwd_launch<5>(B, T, C, x, shift, p, m, out, s);
        case 4: return ddlerp_fwd_launch<4>(B, T, C, x, shift, p, m, out, s);
        case 3: return ddlerp_fwd_launch<3>(B, T, C, x, shift, p, m, out, s);
        default: return ddlerp_fwd_launch<1>(B, T, C, x, shift, p, m, out, s);
    }
}

int wkv_ddlerp_forward(int B, int T, int C, int nmix, const void *x, const void *shift, const float *maa,
                       const void *m, void *out, void *stream) {
    const void *p[5] = {};
    for (int i = 0; i < 5 && i < nmix; i++) p[i] = maa ? maa + (size_t)i * C : nullptr;
    return wkvx_ddlerp_forward(B, T, C, nmix, x, shift, maa ? p : nullptr, WKV_F32, 0, m, out, stream);
}

size_t wkv_ddlerp_backward_workspace(int B, int T, int C, int nmix) {
    if (B <= 0 || T <= 0 || C <= 0) return 0;
    if (!mixes_ok(nmix)) return 0;
    return ddlerp_rows(B, T, C) * nmix * C * sizeof(float);
}

int wkvx_ddlerp_backward(int B, int T, int C, int nmix, const void *x, const void *shift, const void *const *maa, int maa_dtype,
                         int one_minus, const void *m, const void *gout, const void *gshift_in, const void *gx_add,
                         const void *gshift_add, void *gx, void *gm, void *gshift_out, void *const *gmaa, void *workspace,
                         size_t workspace_bytes, void *stream) {
    if (B < 0 || T < 0 || C < 0 || C % 8 != 0) return WKV_ERR_SHAPE;
    if (!mixes_ok(nmix)) return WKV_ERR_UNSUPPORTED;
    if (!gmaa) return WKV_ERR_NULL;
    cudaStream_t s = (cudaStream_t)stream;
    if (B == 0 || T == 0 || C == 0) {
        for (int i = 0; i < nmix && C > 0; i++)
            if (cudaMemsetAsync(gmaa[i], 0, (size_t)C * (maa_dtype == WKV_F32 ? 4 : 2), s) != cudaSuccess) return WKV_ERR_LAUNCH;
        return WKV_OK;
    }
    if (!x || !shift || !maa || !gout || !gx || (m && !gm)) return WKV_ERR_NULL;
    for (int i = 0; i < nmix; i++)
        if (!maa[i]) return WKV_ERR_NULL;
        else if (!aligned16(maa[i])) return WKV_ERR_ALIGN;
    if (!all_aligned({x, shift, m, gout, gshift_in, gx_add, gshift_add, gx, gm, gshift_out})) return WKV_ERR_ALIGN;
    if (!workspace || workspace_bytes < wkv_ddlerp_backward_workspace(B, T, C, nmix)) return WKV_ERR_WORKSPACE;
    const MixPtrs p = mix_ptrs(nmix, maa, maa_dtype, one_minus);
    float *part = (float *)workspace;
    int err;
    switch (nmix) {
        case 5: err = ddlerp_bwd_launch<5>(B, T, C, x, shift, p, m, gout, gshift_in, gx_add, gshift_add, gx, gm, gshift_out, part, s); break;
        case 4: err = ddlerp_bwd_launch<4>(B, T, C, x, shift, p, m, gout, gshift_in, gx_add, gshift_add, gx, gm, gshift_out, part, s); break;
        case 3: err = ddlerp_bwd_launch<3>(B, T, C, x, shift, p, m, gout, gshift_in, gx_add, gshift_add, gx, gm, gshift_out, part, s); break;
        default: err = ddlerp_bwd_launch<1>(B, T, C, x, shift, p, m, gout, gshift_in, gx_add, gshift_add, gx, gm, gshift_out, part, s);
    }
    if (err != WKV_OK) return err;
    return fold_cols(part, ddlerp_rows(B, T, C), nmix, C, gmaa, maa_dtype, one_minus ? -1.f : 1.f, s);
}

int wkv_ddlerp_backward(int B, int T, int C, int nmix, const void *x, const void *shift, const float *maa, const void *m,
                        const void *gout, const void *gshift_in, void *gx, void *gm, void *gshift_out, float *gmaa,
                        void *workspace, size_t workspace_bytes, void *stream) {
    const void *p[5] = {};
    void *g[5] = {};
    for (int i = 0; i < 5 && i < nmix; i++) {
        p[i] = maa ? maa + (size_t)i * C : nullptr;
        g[i] = gmaa ? gmaa + (size_t)i * C : nullptr;
    }
    return wkvx_ddlerp_backward(B, T, C, nmix, x, shift, maa ? p : nullptr, WKV_F32, 0, m, gout, gshift_in, nullptr, nullptr, gx, gm,
                                gshift_out, gmaa ? g : nullptr, workspace, workspace_bytes, stream);
}

}  // extern "C"
