// One token of a time-mix block for a few rows (decode): the block as a short chain of kernels.
//
// With up to 8 rows every projection is a matrix-vector product: the weights (5 C^2 bf16 for v5/v6) are read once and
// everything else is small, so the floor is their HBM time (C = 2560: 65 MB, 10 us) and the enemy is the chain's
// latency: as separate library calls the projections took 8 us each and the block fifteen launches (72 us of GPU
// time, 126 us in all; now 38).  The rows cost shared-memory reads for every output row; how many are taken at which
// width, and what both sides measure, stands at decode_fits() in native_blocks.cpp.  Here:
//
//   v6   strip (x, W1 -> tanh)  ->  mix5 (W2 -> the five mixed inputs)  ->  linear (r, k, v, g and the decay's W1)
//        ->  step (decay, WKV, group norm, silu gate)  ->  linear (output)
//   v5   linear (mixes applied on the way in; r, k, v, g)  ->  step  ->  linear
//
// A warp of `linear` owns one output row per matrix and holds its weights in registers before it waits for the
// kernel ahead (programmatic dependent launch: weights are not written by the chain), so the weight traffic of a kernel
// runs under the latency of the ones before it.  To that end every kernel but the first lets its successor be
// scheduled before its own wait; the first waits before it does, so nothing of the chain runs before the
// work ahead of the block is complete.
//
// Every tensor is rounded to bf16 where the separate operators would store it.
#include "wkv_common.cuh"
#include "wkv_internal.h"

namespace wkv {
namespace {

typedef __nv_bfloat16 bf16;
constexpr float LOG_FLOOR = -5.298317367f;   // log(0.005), as in the chunked WKV kernels

__device__ __forceinline__ float param(const void *p, int dtype, size_t i) {
    return dtype == WKV_F32 ? ((const float *)p)[i] : dtype == WKV_BF16 ? __bfloat162float(((const bf16 *)p)[i]) : __half2float(((const __half *)p)[i]);
}
// tanh to a few fp32 roundings of its value for every x (1 - 2 / (1 + e^{2x}) is that close to 1 only: for small x the
// difference cancels, and under 6e-8 it is zero; low-rank maps start out with such values).  With E = e^{-2|x|} - 1:
// tanh|x| = -E / (2 + E).
__device__ __forceinline__ float tanh_full(float x) {
    const float e = expm1f(-2.f * fabsf(x));
    return copysignf(__fdividef(-e, 2.f + e), x);
}

// x + (shift - x) * maa for 8 channels; one_minus: the parameter is 1 - maa
__device__ __forceinline__ uint4 mix8(const uint4 &x4, const uint4 &s4, const void *maa, int dtype, int one_minus, int c) {
    float x[8], s[8];
    unpack8(x4, x);
    unpack8(s4, s);
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const float a = param(maa, dtype, c + q);
        x[q] += (s[q] - x[q]) * (one_minus ? 1.f - a : a);
    }
    return pack8(x);
}

// out[m][n0..n0+7] = tanh(sum_c x[m][c] W[c][n0..]) for the CTA's 8 columns; x [MT][C] in shared memory (rows past M zero)
template <int MT>
__device__ __forceinline__ void strip(const bf16 *W, int ldw, int n0, const bf16 *xs, int C, int M, bf16 *out) {
    __shared__ float red[8][MT][8];
    float acc[MT][8];
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
        for (int q = 0; q < 8; q++) acc[m][q] = 0.f;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
#pragma unroll 4
    for (int c = tid; c < C; c += 256) {
        float w[8];
        unpack8(*reinterpret_cast<const uint4 *>(W + (size_t)c * ldw + n0), w);
#pragma unroll
        for (int m = 0; m < MT; m++) {
            const float x = __bfloat162float(xs[m * C + c]);
#pragma unroll
            for (int q = 0; q < 8; q++) acc[m][q] = fmaf(x, w[q], acc[m][q]);
        }
    }
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const float s = warp_sum(acc[m][q]);
            if (lane == 0) red[warp][m][q] = s;
        }
    __syncthreads();
    if (tid < MT * 8) {
        const int m = tid >> 3, q = tid & 7;
        float s = 0.f;
#pragma unroll
        for (int g = 0; g < 8; g++) s += red[g][m][q];
        if (m < M) out[(size_t)m * ldw + n0 + q] = __float2bfloat16_rn(tanh_full(bf16_round(s)));
    }
}

// ------------------------------------------------------------------------------ v6: the first low-rank map
struct Strip {
    int M, C, N;                // W [C, N]
    const bf16 *x, *shift;      // [M, C]
    const void *maa;
    int dtype;
    const bf16 *W;
    bf16 *out;                  // [M, N]
    bf16 *new_shift;            // [M, C] copy of x
};
template <int MT>
__global__ void __launch_bounds__(256) k_dec_strip(const Strip P) {
    pdl_wait();
    pdl_trigger();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    bf16 *xs = reinterpret_cast<bf16 *>(smem_raw);
    const int C8 = P.C / 8;
    for (int i = threadIdx.x; i < MT * C8; i += 256) {
        const int m = i / C8, c = (i - m * C8) * 8;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (m < P.M) {
            const uint4 x = *reinterpret_cast<const uint4 *>(P.x + (size_t)m * P.C + c);
            v = mix8(x, *reinterpret_cast<const uint4 *>(P.shift + (size_t)m * P.C + c), P.maa, P.dtype, 0, c);
            if (blockIdx.x == 0) *reinterpret_cast<uint4 *>(P.new_shift + (size_t)m * P.C + c) = x;
        }
        *reinterpret_cast<uint4 *>(xs + m * P.C + c) = v;
    }
    __syncthreads();
    strip<MT>(P.W, P.N, blockIdx.x * 8, xs, P.C, P.M, P.out);
}

// ------------------------------------------------------------------------------ v6: the five mixes
struct Mix5 {
    int M, C;
    const bf16 *x, *shift, *t1, *W2;        // t1 [M, 5, 32]; W2 [5, 32, C]
    const void *maa[5];
    int dtype;
    bf16 *out;                              // [5, M, C]
};
// 32 column chunks of 8 channels x 4 groups of 8 rows of W2
template <int MT>
__global__ void __launch_bounds__(128) k_dec_mix5(const Mix5 P) {
    pdl_trigger();
    __shared__ __align__(16) float part[4][MT][256];
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5, c = (blockIdx.x * 32 + lane) * 8, n = blockIdx.y;
    const bool live = c < P.C;
    uint4 w[8];
#pragma unroll
    for (int j = 0; j < 8; j++)
        w[j] = live ? __ldg(reinterpret_cast<const uint4 *>(P.W2 + ((size_t)n * 32 + g * 8 + j) * P.C + c)) : make_uint4(0u, 0u, 0u, 0u);
    pdl_wait();
    float acc[MT][8];
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
        for (int q = 0; q < 8; q++) acc[m][q] = 0.f;
#pragma unroll
    for (int j = 0; j < 8; j++) {
        float wf[8];
        unpack8(w[j], wf);
#pragma unroll
        for (int m = 0; m < MT; m++) {
            const float t = m < P.M ? __bfloat162float(P.t1[((size_t)m * 5 + n) * 32 + g * 8 + j]) : 0.f;
#pragma unroll
            for (int q = 0; q < 8; q++) acc[m][q] = fmaf(t, wf[q], acc[m][q]);
        }
    }
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
        for (int q = 0; q < 8; q++) part[g][m][lane * 8 + q] = acc[m][q];
    __syncthreads();
    if (!live) return;
    for (int m = g; m < P.M; m += 4) {
        float x[8], s[8];
        unpack8(*reinterpret_cast<const uint4 *>(P.x + (size_t)m * P.C + c), x);
        unpack8(*reinterpret_cast<const uint4 *>(P.shift + (size_t)m * P.C + c), s);
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const int i = lane * 8 + q;
            const float md = bf16_round((part[0][m][i] + part[1][m][i]) + (part[2][m][i] + part[3][m][i]));
            x[q] += (s[q] - x[q]) * (param(P.maa[n], P.dtype, c + q) + md);
        }
        *reinterpret_cast<uint4 *>(P.out + ((size_t)n * P.M + m) * P.C + c) = pack8(x);
    }
}

// ------------------------------------------------------------------------------ matrix-vector products
struct Linear {
    int M, C, n;                // input rows and width; matrices
    const bf16 *W[4];           // [rows, C]
    int rows[4], first[4];      // first: the matrix's first CTA
    bf16 *out[4];               // [M, rows]
    const bf16 *in[4];          // [M, C]: the input of each matrix, or (mix) all x
    int mix, dtype;             // mix: the input is x + (shift - x) * (1 - maa)
    const bf16 *shift;
    const void *maa[4];
    bf16 *new_shift;            // mix: copy of x
    const bf16 *D;              // or NULL: [C, dr], dd = tanh(din D) in the CTAs from dfirst on
    int dr, dfirst;
    const bf16 *din;
    bf16 *dd;
    int chain_head;             // nothing of this chain runs before: wait, then let the successor in
};
// A warp owns one row; its first PRE chunks of 8 weights per lane are in registers before the wait.
template <int MT, int PRE>
__global__ void __launch_bounds__(256) k_dec_linear(const Linear P) {
    if (P.chain_head) pdl_wait();
    pdl_trigger();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    bf16 *xs = reinterpret_cast<bf16 *>(smem_raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, C8 = P.C / 8, cta = blockIdx.x;
    const bool low_rank = P.D && cta >= P.dfirst;
    int mat = 0;
    while (mat + 1 < P.n && cta >= P.first[mat + 1]) mat++;
    const int row = (cta - P.first[mat]) * 8 + warp;
    const bool live = !low_rank && row < P.rows[mat];
    const uint4 *wrow = reinterpret_cast<const uint4 *>(P.W[mat] + (live ? (size_t)row * P.C : 0));
    uint4 w[PRE];
#pragma unroll
    for (int j = 0; j < PRE; j++)
        if (live && lane + 32 * j < C8) w[j] = __ldg(wrow + lane + 32 * j);
    if (!P.chain_head) pdl_wait();
    const bf16 *in = low_rank ? P.din : P.in[mat];
    for (int i = tid; i < MT * C8; i += 256) {
        const int m = i / C8, c = (i - m * C8) * 8;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (m < P.M) {
            v = *reinterpret_cast<const uint4 *>(in + (size_t)m * P.C + c);
            if (P.mix) {
                if (cta == 0) *reinterpret_cast<uint4 *>(P.new_shift + (size_t)m * P.C + c) = v;
                v = mix8(v, *reinterpret_cast<const uint4 *>(P.shift + (size_t)m * P.C + c), P.maa[mat], P.dtype, 1, c);
            }
        }
        *reinterpret_cast<uint4 *>(xs + m * P.C + c) = v;
    }
    __syncthreads();
    if (low_rank) {
        strip<MT>(P.D, P.dr, (cta - P.dfirst) * 8, xs, P.C, P.M, P.dd);
        return;
    }
    if (!live) return;
    float acc[MT];
#pragma unroll
    for (int m = 0; m < MT; m++) acc[m] = 0.f;
    auto chunk = [&](const uint4 &wc, int ch) {
        float wf[8];
        unpack8(wc, wf);
#pragma unroll
        for (int m = 0; m < MT; m++) {
            float xf[8];
            unpack8(*reinterpret_cast<const uint4 *>(xs + m * P.C + ch * 8), xf);
#pragma unroll
            for (int q = 0; q < 8; q++) acc[m] = fmaf(wf[q], xf[q], acc[m]);
        }
    };
#pragma unroll
    for (int j = 0; j < PRE; j++)
        if (lane + 32 * j < C8) chunk(w[j], lane + 32 * j);
#pragma unroll 2
    for (int ch = lane + 32 * PRE; ch < C8; ch += 32) chunk(__ldg(wrow + ch), ch);
#pragma unroll
    for (int m = 0; m < MT; m++) {
        const float s = warp_sum(acc[m]);
        if (lane == 0 && m < P.M) P.out[mat][(size_t)m * P.rows[mat] + row] = __float2bfloat16_rn(s);
    }
}

// ------------------------------------------------------------------------------ v5 / v6: WKV step, group norm, gate
struct Step {
    int M, H;
    const bf16 *r, *k, *v, *g;      // [M, C]
    const void *u;                  // [H, 64] bf16
    const bf16 *dd, *D2;            // v6: [M, dr], [dr, C]
    int dr;
    const void *decay;              // v6: [C] bf16;  v5: time_decay [C]
    int decay_dtype;
    const void *lw, *lb;            // group norm
    int ln_dtype;
    float eps;
    const float *s0;                // [M, H, 64, 64] (key, value)
    float *s1;
    bf16 *out;                      // [M, C] norm(y) * silu(g)
};
// One CTA per (row, head): thread = 4 value columns x 4 key rows (of 16 groups).
template <bool V6>
__global__ void __launch_bounds__(256) k_dec_step(const Step P) {
    pdl_trigger();
    __shared__ float sr[64], sk[64], sw[64], su[64], wpart[4][64], red[4];
    __shared__ __align__(16) float part[16][64];
    const int m = blockIdx.x / P.H, h = blockIdx.x - m * P.H, C = P.H * 64, tid = threadIdx.x, c = tid & 63, g4 = tid >> 6;
    const int col = (tid & 15) * 4, rg = tid >> 4;
    const float *s0 = P.s0 + (size_t)blockIdx.x * 4096;
    pdl_wait();
    float4 S[4];
#pragma unroll
    for (int i = 0; i < 4; i++) S[i] = *reinterpret_cast<const float4 *>(s0 + (rg * 4 + i) * 64 + col);
    const size_t at = (size_t)m * C + h * 64 + c;
    if (g4 == 0) { sr[c] = __bfloat162float(P.r[at]); su[c] = __bfloat162float(((const bf16 *)P.u)[h * 64 + c]); }
    if (g4 == 1) sk[c] = __bfloat162float(P.k[at]);
    if (V6) {
        // the decay's second low-rank map: 64 channels x 4 groups of rows
        float a = 0.f;
        const int n = P.dr / 4;
#pragma unroll 8
        for (int j = g4 * n; j < g4 * n + n; j++)
            a = fmaf(__bfloat162float(P.dd[(size_t)m * P.dr + j]), __bfloat162float(P.D2[(size_t)j * C + h * 64 + c]), a);
        wpart[g4][c] = a;
    }
    __syncthreads();
    if (g4 == 0) {
        float x;
        if (V6) x = bf16_round(param(P.decay, P.decay_dtype, h * 64 + c) + ((wpart[0][c] + wpart[1][c]) + (wpart[2][c] + wpart[3][c])));
        else x = param(P.decay, P.decay_dtype, h * 64 + c);
        sw[c] = __expf(fmaxf(-__expf(x), LOG_FLOOR));
    }
    __syncthreads();
    const uint2 v4 = *reinterpret_cast<const uint2 *>(P.v + (size_t)m * C + h * 64 + col);
    const float vv[4] = {__uint_as_float(v4.x << 16), __uint_as_float(v4.x & 0xFFFF0000u), __uint_as_float(v4.y << 16), __uint_as_float(v4.y & 0xFFFF0000u)};
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    float *s1 = P.s1 + (size_t)blockIdx.x * 4096;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int row = rg * 4 + i;
        const float r = sr[row], k = sk[row], w = sw[row], b = r * su[row] * k;
        float *s = reinterpret_cast<float *>(&S[i]);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            acc[q] = fmaf(r, s[q], fmaf(b, vv[q], acc[q]));
            s[q] = fmaf(w, s[q], k * vv[q]);
        }
        *reinterpret_cast<float4 *>(s1 + row * 64 + col) = S[i];
    }
    *reinterpret_cast<float4 *>(&part[rg][col]) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    __syncthreads();
    if (tid < 64) {
        float y = 0.f;
#pragma unroll
        for (int j = 0; j < 16; j++) y += part[j][c];
        y = bf16_round(y);
        // the 64 channels sit in two warps
        const float s = warp_sum(y);
        if ((tid & 31) == 0) red[tid >> 5] = s;
        asm volatile("bar.sync 1, 64;" ::: "memory");
        const float d = y - (red[0] + red[1]) * (1.f / 64.f), v = warp_sum(d * d);
        if ((tid & 31) == 0) red[2 + (tid >> 5)] = v;
        asm volatile("bar.sync 1, 64;" ::: "memory");
        const float rstd = rsqrtf((red[2] + red[3]) * (1.f / 64.f) + P.eps), gr = __bfloat162float(P.g[at]);
        const float o = d * rstd * param(P.lw, P.ln_dtype, h * 64 + c) + param(P.lb, P.ln_dtype, h * 64 + c);
        P.out[at] = __float2bfloat16_rn(o * bf16_round(gr * sigmoidf(gr)));
    }
}

constexpr int MAX_SMEM = 200 * 1024;
template <int MT>
int strip_launch(const Strip &P, cudaStream_t s) {
    static unsigned char done[64];
    if (!set_max_smem_once(k_dec_strip<MT>, MAX_SMEM, done)) return WKV_ERR_LAUNCH;
    return launch_chained(k_dec_strip<MT>, dim3(P.N / 8), dim3(256), (size_t)MT * P.C * 2, s, P);
}
template <int MT>
int linear_launch(const Linear &P, int ctas, cudaStream_t s) {
    // 10 chunks of 8 x 32 weights: rows of up to 2560 are prefetched whole, wider rows stream the rest.  One row, us with 3 / 6 /
    // 10 / 16 chunks ahead: v6 C = 768 19.4 / 19.5 / 19.4 / 20.8, C = 2560 38.3 / 36.8 / 36.6 / 41.7, C = 4096 59.3 / 57.7 / 62.5 /
    // 60.9; v5 8.9 / 9.0 / 9.4 / 11.1, 27.3 / 25.7 / 23.7 / 31.0, 46.3 / 44.5 / 51.6 / 47.8.  (A row that does not fit is better off with
    // 6: registers it cannot use up cost warps.)
    static unsigned char done[64];
    if (!set_max_smem_once(k_dec_linear<MT, 10>, MAX_SMEM, done)) return WKV_ERR_LAUNCH;
    return launch_chained(k_dec_linear<MT, 10>, dim3(ctas), dim3(256), (size_t)MT * P.C * 2, s, P);
}
template <int MT>
int mix5_launch(const Mix5 &P, cudaStream_t s) {
    return launch_chained(k_dec_mix5<MT>, dim3((P.C / 8 + 31) / 32, 5), dim3(128), 0, s, P);
}
int linear(Linear &P, cudaStream_t s) {
    int ctas = 0;
    for (int i = 0; i < P.n; i++) {
        P.first[i] = ctas;
        ctas += (P.rows[i] + 7) / 8;
    }
    P.dfirst = ctas;
    if (P.D) ctas += P.dr / 8;
    return P.M == 1 ? linear_launch<1>(P, ctas, s) : P.M == 2 ? linear_launch<2>(P, ctas, s) : P.M <= 4 ? linear_launch<4>(P, ctas, s) : linear_launch<8>(P, ctas, s);
}

}  // namespace
}  // namespace wkv

using namespace wkv;

extern "C" {

int wkvx_decode_max_rows(void) { return 8; }

int wkvx_decode6(const wkvx_decode6_t *a, void *stream) {
    if (!a || a->M < 1 || a->M > 8 || a->H < 1 || a->H > 128 || a->rank != 32 || a->decay_rank % 8) return WKV_ERR_SHAPE;
    if (!all_aligned({a->x, a->shift, a->w1, a->w2, a->d1, a->proj[0], a->proj[1], a->proj[2], a->proj[3], a->proj[4], a->state_in, a->xs, a->rkvg,
                      a->normed, a->new_shift, a->state_out}))
        return WKV_ERR_ALIGN;
    const int M = a->M, C = a->H * 64;
    cudaStream_t s = (cudaStream_t)stream;
    typedef const __nv_bfloat16 *cb;
    typedef __nv_bfloat16 *mb;
    Strip st{M, C, 5 * a->rank, (cb)a->x, (cb)a->shift, a->maa_x, a->maa_dtype, (cb)a->w1, (mb)a->t1, (mb)a->new_shift};
    int err = M == 1 ? strip_launch<1>(st, s) : M == 2 ? strip_launch<2>(st, s) : M <= 4 ? strip_launch<4>(st, s) : strip_launch<8>(st, s);
    if (err != WKV_OK) return err;
    Mix5 mx{M, C, (cb)a->x, (cb)a->shift, (cb)a->t1, (cb)a->w2, {}, a->maa_dtype, (mb)a->xs};
    for (int i = 0; i < 5; i++) mx.maa[i] = a->maa[i];
    err = M == 1 ? mix5_launch<1>(mx, s) : M == 2 ? mix5_launch<2>(mx, s) : M <= 4 ? mix5_launch<4>(mx, s) : mix5_launch<8>(mx, s);
    if (err != WKV_OK) return err;
    // mixed inputs in the order w, k, v, r, g
    cb xs = (cb)a->xs;
    mb rkvg = (mb)a->rkvg;
    const size_t n = (size_t)M * C;
    Linear L = {};
    L.M = M; L.C = C; L.n = 4;
    const int order[4] = {3, 1, 2, 4};
    for (int i = 0; i < 4; i++) {
        L.W[i] = (cb)a->proj[i];
        L.rows[i] = C;
        L.out[i] = rkvg + i * n;
        L.in[i] = xs + order[i] * n;
    }
    L.D = (cb)a->d1; L.dr = a->decay_rank; L.din = xs; L.dd = (mb)a->dd;
    err = linear(L, s);
    if (err != WKV_OK) return err;
    Step sp = {M, a->H, rkvg, rkvg + n, rkvg + 2 * n, rkvg + 3 * n, a->u, (cb)a->dd, (cb)a->d2, a->decay_rank, a->decay, WKV_BF16, a->ln_w, a->ln_b,
               a->ln_dtype, a->eps, a->state_in, a->state_out, (mb)a->normed};
    err = launch_chained(k_dec_step<true>, dim3(M * a->H), dim3(256), 0, s, sp);
    if (err != WKV_OK) return err;
    Linear O = {};
    O.M = M; O.C = C; O.n = 1;
    O.W[0] = (cb)a->proj[4]; O.rows[0] = C; O.out[0] = (mb)a->out; O.in[0] = (cb)a->normed;
    return linear(O, s);
}

int wkvx_decode5(const wkvx_decode5_t *a, void *stream) {
    if (!a || a->M < 1 || a->M > 8 || a->H < 1 || a->H > 128 || a->C < 8 || a->C % 8 || a->C > 8192) return WKV_ERR_SHAPE;
    if (!all_aligned({a->x, a->shift, a->proj[0], a->proj[1], a->proj[2], a->proj[3], a->proj[4], a->state_in, a->rkvg, a->normed, a->new_shift,
                      a->state_out}))
        return WKV_ERR_ALIGN;
    const int M = a->M, A = a->H * 64;
    cudaStream_t s = (cudaStream_t)stream;
    typedef const __nv_bfloat16 *cb;
    typedef __nv_bfloat16 *mb;
    mb rkvg = (mb)a->rkvg;
    const size_t n = (size_t)M * A;
    Linear L = {};
    L.M = M; L.C = a->C; L.n = 4; L.mix = 1; L.dtype = a->mix_dtype; L.shift = (cb)a->shift; L.new_shift = (mb)a->new_shift; L.chain_head = 1;
    const int order[4] = {2, 0, 1, 3};      // mixes in the order k, v, r, g
    for (int i = 0; i < 4; i++) {
        L.W[i] = (cb)a->proj[i];
        L.rows[i] = A;
        L.out[i] = rkvg + i * n;
        L.in[i] = (cb)a->x;
        L.maa[i] = a->mix[order[i]];
    }
    int err = linear(L, s);
    if (err != WKV_OK) return err;
    Step sp = {M, a->H, rkvg, rkvg + n, rkvg + 2 * n, rkvg + 3 * n, a->u, nullptr, nullptr, 0, a->decay, a->decay_dtype, a->ln_w, a->ln_b, a->ln_dtype, a->eps,
               a->state_in, a->state_out, (mb)a->normed};
    err = launch_chained(k_dec_step<false>, dim3(M * a->H), dim3(256), 0, s, sp);
    if (err != WKV_OK) return err;
    Linear O = {};
    O.M = M; O.C = A; O.n = 1;
    O.W[0] = (cb)a->proj[4]; O.rows[0] = a->C; O.out[0] = (mb)a->out; O.in[0] = (cb)a->normed;
    return linear(O, s);
}

}  // extern "C"
