// Token-serial fp32 kernels for the v5/v6 WKV recurrence (any element type, any T): the exact path
// behind the fp32 and fp16 entry points, and the forward path of bf16 calls of a few tokens (decode).
//
// The 64x64 state of a (batch, head) lives in registers and a token is two fused multiply-adds and one
// multiply per element.  Everything else is kept off that chain: one warp of every CTA loads the tokens,
// exponentiates the decays, forms the per-token scalar and stages tiles of TT tokens in shared memory, STAGES
// ahead of the warps that hold the state, and no token waits for the reduction of the one before.  Two
// shapes of the same step:
//
//   column   M[:,v]: out[v] = sum_k a_k M[k,v] + bonus x_v;    M[k,v] = w_k M[k,v] + d_k x_v
//            forward   (t up):   a = r, d = k, x = v,  out = y        bonus = sum_k r_k u_k k_k
//            role C    (t down): a = k, d = r, x = gy, out = gv       (the same bonus)
//   row      M[k,:]: out[k] = sum_v a_v M[k,v] + u_k d_k g;    M[k,v] = w_k M[k,v] + d_k x_v
//            role A    (t up):   a = gy, d = k, x = v,  out = gr      g = sum_v v_v gy_v
//            role B    (t down): a = v,  d = r, x = gy, out = gk
//
// Backward runs the roles A, B and C side by side in one launch (they carry S, D and D and need nothing from
// one another), then k_serial_gw for the decay gradient from what A and B leave per token,
//   q_t[k] = r_t[k] sum_v S_t[k,v] gy_t[v],   p_t[k] = k_t[k] sum_v D_{t+1}[k,v] v_t[v]:
//   E_t = E_{t+1} + q_t - p_t,  E_T = sum_v S_T[k,v] D_T[k,v],   dL/d(log w_t) = E_{t+1} - p_t.
//
// A warp holds 4 x 16 elements of the reduced dimension by 8*NC of the other (thread: 16 x NC).  What bounds
// it is the SM's shared-memory port: an LDS.128 takes 4 of its cycles whatever it broadcasts, so a
// column-shaped warp needs 48 of them per token for NC = 1 and for NC = 4 alike.  Few heads: NC = 1, eight
// one-warp CTAs a head, the shortest chain.  Many: NC = 4, two warps a head, a quarter of the port time.
// Unrolling a token more than this makes it slower (a lone warp then waits for instructions), a second loading
// warp too.  fp32, 8 heads, 128 tokens: forward 78 -> 12 us, backward 141 -> 26 us against two barriers and an
// exposed load per token; bf16 decode (T = 1), 512 heads: 4 us instead of 35 us on the chunked kernel.
// Same math as RWKV-v5/src/module/cuda/wkv5_cuda.cu:129-340 and
// RWKV-v6/src/module/cuda/wkv6state_cuda_v1.cu:6-293, plus what those lack:
// per-batch state, state_out, gstate_out -> gstate_in.
#include "wkv_common.cuh"

namespace wkv {
namespace {

constexpr int N = HEAD;
constexpr int TT = 8;             // tokens per staged tile
constexpr int STAGES = 4;
constexpr float LOG_FLOOR = -5.298317367f;   // log(0.005), the floor of the chunked kernels

// where the log-decay (<= 0) comes from: v5's fp32 [H,64] in either encoding, v6's per-token activation x
// (element type F), v6's per-token fp32 ew = -exp(x)
enum { W_STATIC = 0, W_X = 1, W_EW = 2 };
template <typename F, int WSRC> struct WElem { typedef F type; };
template <typename F> struct WElem<F, W_EW> { typedef float type; };
template <typename F, int WSRC>
__device__ __forceinline__ float log_decay(typename WElem<F, WSRC>::type w) {
    const float x = Elem<typename WElem<F, WSRC>::type>::ld(&w);
    return WSRC == W_X ? -expf(x) : x;
}
__device__ __forceinline__ float static_log_decay(const void *w, int w_kind, int c) {
    const float x = ((const float *)w)[c];
    return w_kind == WKV_W_RAW ? -expf(x) : x;
}

__device__ __forceinline__ size_t state_idx(int layout, int key, int val) {
    return layout == WKV_STATE_KV ? (size_t)key * N + val : (size_t)val * N + key;
}

struct SerialParams {
    int T, H, w_kind, layout, floor;    // (w_kind: W_STATIC alone)
    const void *r, *k, *v, *w, *u, *gy;
    const float *s0, *g0;       // state_in, gstate_out (or NULL)
    void *y;                    // forward
    float *s1;                  // state_out
    void *gr, *gk, *gv;         // backward
    float *g1;                  // gstate_in
    float *q, *p, *eT;          // [B,T,C], [B,T,C], [B,C]
    float *gu;                  // [B,C]
};

// Staged vectors of a tile: a (read-out) and x-side / d-side vectors, decays.
struct __align__(16) Stage {
    float a[TT][N], d[TT][N], w[TT][N], x[TT][N];
    float m[TT][N];             // row roles: what the reduced value is multiplied by for q / p
    float dot[TT];              // the per-token scalar (bonus / g)
};

// Hand-over of a stage between the loading warp that fills it and the CW state warps, on named barriers 1 + 2 * stage
// (full) and 2 + 2 * stage (empty): one side arrives, the other waits.
template <int CW> __device__ __forceinline__ void bar_arrive(int id) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(32 * (CW + 1)) : "memory");
}
template <int CW> __device__ __forceinline__ void bar_wait(int id) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(32 * (CW + 1)) : "memory");
}

template <typename F> struct Two;      // two adjacent elements, loaded together
template <> struct Two<float> { typedef float2 raw; static __device__ __forceinline__ float2 f(float2 v) { return v; } };
template <> struct Two<__nv_bfloat16> {
    typedef __nv_bfloat162 raw;
    static __device__ __forceinline__ float2 f(__nv_bfloat162 v) { return __bfloat1622float2(v); }
};
template <> struct Two<__half> {
    typedef __half2 raw;
    static __device__ __forceinline__ float2 f(__half2 v) { return __half22float2(v); }
};

// element (i of 16, n of NC) of the state: reduced index 16*(i/4) + 4*q + i%4, other index o0 + n
__device__ __forceinline__ int red_index(int i, int q) { return 16 * (i >> 2) + 4 * q + (i & 3); }

// Sum over the four lanes q.  Afterwards lane q holds the total of entry own_entry(q); the lanes with
// owns(q) hold every entry once.
template <int NC> __device__ __forceinline__ int own_entry(int q) { return NC == 4 ? q : NC == 2 ? q >> 1 : 0; }
template <int NC> __device__ __forceinline__ bool owns(int q) { return NC == 4 || (NC == 2 ? !(q & 1) : q == 0); }
template <int NC>
__device__ __forceinline__ float reduce_q(float (&acc)[NC], int q) {
    if constexpr (NC == 4) {
        const bool b1 = q & 2, b0 = q & 1;
        const float s0 = b1 ? acc[0] : acc[2], s1 = b1 ? acc[1] : acc[3];
        float k0 = (b1 ? acc[2] : acc[0]) + __shfl_xor_sync(0xffffffffu, s0, 16);
        float k1 = (b1 ? acc[3] : acc[1]) + __shfl_xor_sync(0xffffffffu, s1, 16);
        return (b0 ? k1 : k0) + __shfl_xor_sync(0xffffffffu, b0 ? k0 : k1, 8);
    } else {
        float v;
        if constexpr (NC == 2) v = (q & 2 ? acc[1] : acc[0]) + __shfl_xor_sync(0xffffffffu, q & 2 ? acc[0] : acc[1], 16);
        else v = acc[0] + __shfl_xor_sync(0xffffffffu, acc[0], 16);
        return v + __shfl_xor_sync(0xffffffffu, v, 8);
    }
}

// The state of a thread to / from global memory.  COLUMN: reduced index = key, other = value; else the reverse.
template <bool COLUMN, int NC>
__device__ __forceinline__ void load_state(float (&M)[16][NC], const float *s, int layout, int q, int o0) {
    // along whichever index the layout keeps contiguous: the reduced one (quads of i) or the other one (n)
    const bool along_red = (layout == WKV_STATE_KV) != COLUMN;
    if (along_red) {
#pragma unroll
        for (int n = 0; n < NC; n++)
#pragma unroll
            for (int i4 = 0; i4 < 4; i4++) {
                const float4 f = *reinterpret_cast<const float4 *>(s + (size_t)(o0 + n) * N + 16 * i4 + 4 * q);
                M[4 * i4][n] = f.x; M[4 * i4 + 1][n] = f.y; M[4 * i4 + 2][n] = f.z; M[4 * i4 + 3][n] = f.w;
            }
    } else {
#pragma unroll
        for (int i = 0; i < 16; i++) {
            if constexpr (NC == 4) {
                const float4 f = *reinterpret_cast<const float4 *>(s + (size_t)red_index(i, q) * N + o0);
                M[i][0] = f.x; M[i][1] = f.y; M[i][2] = f.z; M[i][3] = f.w;
            } else {
#pragma unroll
                for (int n = 0; n < NC; n++) M[i][n] = s[(size_t)red_index(i, q) * N + o0 + n];
            }
        }
    }
}
template <bool COLUMN, int NC>
__device__ __forceinline__ void store_state(const float (&M)[16][NC], float *s, int layout, int q, int o0) {
    const bool along_red = (layout == WKV_STATE_KV) != COLUMN;
    if (along_red) {
#pragma unroll
        for (int n = 0; n < NC; n++)
#pragma unroll
            for (int i4 = 0; i4 < 4; i4++)
                *reinterpret_cast<float4 *>(s + (size_t)(o0 + n) * N + 16 * i4 + 4 * q) =
                    make_float4(M[4 * i4][n], M[4 * i4 + 1][n], M[4 * i4 + 2][n], M[4 * i4 + 3][n]);
    } else {
#pragma unroll
        for (int i = 0; i < 16; i++) {
            if constexpr (NC == 4)
                *reinterpret_cast<float4 *>(s + (size_t)red_index(i, q) * N + o0) = make_float4(M[i][0], M[i][1], M[i][2], M[i][3]);
            else
#pragma unroll
                for (int n = 0; n < NC; n++) s[(size_t)red_index(i, q) * N + o0 + n] = M[i][n];
        }
    }
}

// One role over the tokens of one (batch, head).  UP: t ascending, else descending.
template <typename F, int WSRC, int NC, int CW, bool COLUMN, bool UP>
__device__ __forceinline__ void
serial_role(const SerialParams &P, Stage (&stage)[STAGES], const F *a_, const F *d_, const F *x_, const F *m_, F *out_,
            const float *init, float *final_state, float *pq) {
    constexpr int PER_CTA = 8 * NC * CW, PER_HEAD = N / PER_CTA;     // other-side indices of a CTA; CTAs of a head
    const int bh = blockIdx.x / PER_HEAD, slice = blockIdx.x - bh * PER_HEAD;
    const int b = bh / P.H, h = bh - b * P.H, C = P.H * N, T = P.T;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ntile = (T + TT - 1) / TT;
    const size_t base = (size_t)b * T * C + (size_t)h * N, sbase = (size_t)bh * N * N;

    if (warp == CW) {
        // ---- the loading warp: two channels a lane.  A tile in flight is kept as loaded (a conversion would
        // wait for the load); tokens past the end read the last one again and count for nothing.
        typedef typename Two<F>::raw R2;
        typedef typename Two<typename WElem<F, WSRC>::type>::raw W2;
        const int c = 2 * lane;
        // (u may start at any element: two loads)
        const float2 u2 = make_float2(Elem<F>::ld((const F *)P.u + h * N + c), Elem<F>::ld((const F *)P.u + h * N + c + 1));
        float ws[2] = {0.f, 0.f};
        if (WSRC == W_STATIC) {
#pragma unroll
            for (int e = 0; e < 2; e++) {
                float lw = static_log_decay(P.w, P.w_kind, h * N + c + e);
                if (P.floor) lw = fmaxf(lw, LOG_FLOOR);
                ws[e] = expf(lw);
            }
        }
        R2 fa[TT], fd[TT], fx[TT], fm[TT];
        W2 fw[TT];
        auto fetch = [&](int tile) {
#pragma unroll
            for (int j = 0; j < TT; j++) {
                const int s = min(tile * TT + j, T - 1), t = UP ? s : T - 1 - s;
                const size_t o = base + (size_t)t * C + c;
                fa[j] = *reinterpret_cast<const R2 *>(a_ + o);
                fd[j] = *reinterpret_cast<const R2 *>(d_ + o);
                fx[j] = *reinterpret_cast<const R2 *>(x_ + o);
                if (!COLUMN) fm[j] = *reinterpret_cast<const R2 *>(m_ + o);
                if (WSRC != W_STATIC)
                    fw[j] = *reinterpret_cast<const W2 *>((const typename WElem<F, WSRC>::type *)P.w + o);
            }
        };
        if (ntile > 0) fetch(0);
        int st = 0;
        for (int tile = 0; tile < ntile; tile++) {
            Stage &S = stage[st];
            if (tile >= STAGES) bar_wait<CW>(2 + 2 * st);
#pragma unroll
            for (int j = 0; j < TT; j++) {
                float2 w = make_float2(ws[0], ws[1]);
                if (WSRC != W_STATIC) {
                    w = Two<typename WElem<F, WSRC>::type>::f(fw[j]);
                    if (WSRC == W_X) { w.x = -expf(w.x); w.y = -expf(w.y); }
                    if (P.floor) { w.x = fmaxf(w.x, LOG_FLOOR); w.y = fmaxf(w.y, LOG_FLOOR); }
                    w.x = expf(w.x); w.y = expf(w.y);
                }
                const float2 a = Two<F>::f(fa[j]), d = Two<F>::f(fd[j]), x = Two<F>::f(fx[j]);
                *reinterpret_cast<float2 *>(&S.a[j][c]) = a;
                *reinterpret_cast<float2 *>(&S.d[j][c]) = d;
                *reinterpret_cast<float2 *>(&S.x[j][c]) = x;
                *reinterpret_cast<float2 *>(&S.w[j][c]) = w;
                if (!COLUMN) *reinterpret_cast<float2 *>(&S.m[j][c]) = Two<F>::f(fm[j]);
                // COLUMN: sum_k a u d (r u k in either order);  row: sum_v a x  (gy v in either order)
                const float s = warp_sum(COLUMN ? a.x * u2.x * d.x + a.y * u2.y * d.y : a.x * x.x + a.y * x.y);
                if (lane == 0) S.dot[j] = s;
            }
            bar_arrive<CW>(1 + 2 * st);
            if (tile + 1 < ntile) fetch(tile + 1);
            st = (st + 1) & (STAGES - 1);
        }
        return;
    }

    // ---- the state warps
    const int q = lane >> 3, cl = lane & 7;
    const int o0 = slice * PER_CTA + (warp * 8 + cl) * NC;     // first of this thread's NC other-side indices
    const int oq = o0 + own_entry<NC>(q);                      // the one whose output it writes
    const float u_o = COLUMN ? 0.f : Elem<F>::ld((const F *)P.u + h * N + oq);
    float M[16][NC];
    if (init) {
        load_state<COLUMN, NC>(M, init + sbase, P.layout, q, o0);
    } else {
#pragma unroll
        for (int i = 0; i < 16; i++)
#pragma unroll
            for (int n = 0; n < NC; n++) M[i][n] = 0.f;
    }
    float gu_acc = 0.f;
    auto token = [&](const Stage &S, int j, int t) {
        constexpr int NA = NC == 1 ? 4 : 1;      // independent partial sums of the reduction
        float acc[NA][NC], drv[NC], dec[NC];
#pragma unroll
        for (int n = 0; n < NC; n++) {
#pragma unroll
            for (int e = 0; e < NA; e++) acc[e][n] = 0.f;
            drv[n] = COLUMN ? S.x[j][o0 + n] : S.d[j][o0 + n];
            dec[n] = COLUMN ? 0.f : S.w[j][o0 + n];
        }
#pragma unroll
        for (int i4 = 0; i4 < 4; i4++) {
            const int at = 16 * i4 + 4 * q;
            const float4 a4 = *reinterpret_cast<const float4 *>(&S.a[j][at]);
            const float4 v4 = *reinterpret_cast<const float4 *>(COLUMN ? &S.d[j][at] : &S.x[j][at]);
            float4 w4 = make_float4(0.f, 0.f, 0.f, 0.f);
            if (COLUMN) w4 = *reinterpret_cast<const float4 *>(&S.w[j][at]);
            const float av[4] = {a4.x, a4.y, a4.z, a4.w}, vv[4] = {v4.x, v4.y, v4.z, v4.w}, wv[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
            for (int e = 0; e < 4; e++)
#pragma unroll
                for (int n = 0; n < NC; n++) {
                    float &m = M[4 * i4 + e][n];
                    acc[NA == 4 ? e : 0][n] = fmaf(av[e], m, acc[NA == 4 ? e : 0][n]);
                    m = fmaf(COLUMN ? wv[e] : dec[n], m, vv[e] * drv[n]);
                }
        }
        if constexpr (NA == 4) acc[0][0] = (acc[0][0] + acc[1][0]) + (acc[2][0] + acc[3][0]);
        const float tot = reduce_q<NC>(acc[0], q);
        const float dot = S.dot[j];
        if (owns<NC>(q)) {
            const size_t o = base + (size_t)t * C + oq;
            if (COLUMN) {
                Elem<F>::st(out_ + o, fmaf(dot, S.x[j][oq], tot));
            } else {
                const float d = S.d[j][oq];
                Elem<F>::st(out_ + o, fmaf(u_o * d, dot, tot));
                // A: q = r * (S gy), and gu's share r k g;   B: p = k * (D v)
                const float m = S.m[j][oq];
                pq[o] = m * tot;
                if (UP) gu_acc = fmaf(m * d, dot, gu_acc);
            }
        }
    };
    int st = 0;
    for (int tile = 0; tile < ntile; tile++) {
        const Stage &S = stage[st];
        bar_wait<CW>(1 + 2 * st);
        const int s0 = tile * TT;
        if (s0 + TT <= T) {
#pragma unroll(NC == 1 ? 4 : 2)
            for (int j = 0; j < TT; j++) token(S, j, UP ? s0 + j : T - 1 - s0 - j);
        } else {
#pragma unroll 1
            for (int j = 0; j < T - s0; j++) token(S, j, UP ? s0 + j : T - 1 - s0 - j);
        }
        if (tile + STAGES < ntile) bar_arrive<CW>(2 + 2 * st);
        st = (st + 1) & (STAGES - 1);
    }
    if (COLUMN) {
        if (final_state) store_state<COLUMN, NC>(M, final_state + sbase, P.layout, q, o0);
    } else if (UP) {
        // E_T = sum_v S_T D_T per key row
        float acc[NC];
#pragma unroll
        for (int n = 0; n < NC; n++) acc[n] = 0.f;
        if (P.g0) {
            float D[16][NC];
            load_state<COLUMN, NC>(D, P.g0 + sbase, P.layout, q, o0);
#pragma unroll
            for (int i = 0; i < 16; i++)
#pragma unroll
                for (int n = 0; n < NC; n++) acc[n] = fmaf(M[i][n], D[i][n], acc[n]);
        }
        const float e = reduce_q<NC>(acc, q);
        if (owns<NC>(q)) {
            P.eT[(size_t)b * C + h * N + oq] = e;
            P.gu[(size_t)b * C + h * N + oq] = gu_acc;
        }
    }
}

template <typename F, int WSRC, int NC, int CW>
__global__ void __launch_bounds__(32 * (CW + 1)) k_serial_fwd(const SerialParams P) {
    pdl_wait();
    pdl_trigger();
    __shared__ Stage stage[STAGES];
    serial_role<F, WSRC, NC, CW, true, true>(P, stage, (const F *)P.r, (const F *)P.k, (const F *)P.v, (const F *)nullptr, (F *)P.y, P.s0, P.s1, nullptr);
}

template <typename F, int WSRC, int NC, int CW>
__global__ void __launch_bounds__(32 * (CW + 1)) k_serial_bwd(const SerialParams P) {
    pdl_wait();
    pdl_trigger();
    __shared__ Stage stage[STAGES];
    const F *r = (const F *)P.r, *k = (const F *)P.k, *v = (const F *)P.v, *gy = (const F *)P.gy;
    if (blockIdx.y == 0) serial_role<F, WSRC, NC, CW, false, true>(P, stage, gy, k, v, r, (F *)P.gr, P.s0, nullptr, P.q);
    else if (blockIdx.y == 1) serial_role<F, WSRC, NC, CW, false, false>(P, stage, v, r, gy, k, (F *)P.gk, P.g0, nullptr, P.p);
    else serial_role<F, WSRC, NC, CW, true, false>(P, stage, k, r, gy, (const F *)nullptr, (F *)P.gv, P.g0, P.g1, nullptr);
}

// Decay gradient: one CTA per (batch, head), 64 channels x 16 groups of consecutive tokens.  Every group sums
// its q - p, the groups' suffix sums meet in shared memory, and a second walk (from L2) gives E_{t+1} - p_t.
template <typename F, int WSRC>
__global__ void __launch_bounds__(1024) k_serial_gw(const SerialParams P, void *gw_out) {
    pdl_wait();
    pdl_trigger();
    __shared__ float tot[16][N];
    const int bh = blockIdx.x, b = bh / P.H, h = bh - b * P.H, C = P.H * N, T = P.T;
    const int c = threadIdx.x & (N - 1), g = threadIdx.x >> 6;
    const int len = (T + 15) / 16, t0 = min(T, g * len), t1 = min(T, t0 + len);
    const size_t base = (size_t)b * T * C + (size_t)h * N + c;
    float s = 0.f;
#pragma unroll 8
    for (int t = t1 - 1; t >= t0; t--) s += P.q[base + (size_t)t * C] - P.p[base + (size_t)t * C];
    tot[g][c] = s;
    __syncthreads();
    float E = P.eT[(size_t)b * C + h * N + c];
    for (int j = 15; j > g; j--) E += tot[j][c];
    float sum = 0.f;
    const float lw_static = WSRC == W_STATIC ? static_log_decay(P.w, P.w_kind, h * N + c) : 0.f;
#pragma unroll 8
    for (int t = t1 - 1; t >= t0; t--) {
        const size_t o = base + (size_t)t * C;
        const float p = P.p[o];
        // (d/dx of log w = -exp(x) is log w)
        if (WSRC != W_STATIC)
            Elem<F>::st((F *)gw_out + o, (E - p) * log_decay<F, WSRC>(((const typename WElem<F, WSRC>::type *)P.w)[o]));
        else sum += E - p;
        E += P.q[o] - p;
    }
    if (WSRC == W_STATIC) {
        __syncthreads();
        tot[g][c] = sum;
        __syncthreads();
        if (g == 0) {
#pragma unroll
            for (int j = 1; j < 16; j++) sum += tot[j][c];
            ((float *)gw_out)[(size_t)b * C + h * N + c] = sum * lw_static;
        }
    }
}

SerialParams make_params(const wkv_args_t *a) {
    SerialParams P = {};
    P.T = a->T; P.H = a->H; P.w_kind = a->w_kind; P.layout = a->state_layout;
    P.r = a->r; P.k = a->k; P.v = a->v; P.w = a->w; P.u = a->u; P.gy = a->gy;
    P.s0 = a->state_in; P.g0 = a->gstate_out;
    P.y = a->y; P.s1 = a->state_out;
    P.gr = a->gr; P.gk = a->gk; P.gv = a->gv; P.g1 = a->gstate_in;
    P.gu = a->gu;
    return P;
}

// Which shape, from the heads x rows the SMs get: with one-warp CTAs of NC = 1 a chain costs the SM's shared-memory port
// 8 x 48 cycles a token, with NC = 2 half, with NC = 4 a quarter; alone, they take about 100, 130 and 250 cycles a token.
// Measured, us for the shapes 1 / 2 / 4:
//   forward, 128 tokens fp32   37 heads 14.0 / 19.8 / 33.1     74: 20.7 / 20.0 / 33.2    100: 37.7 / 28.9 / 33.2
//                             256: 76.0 / 35.6 / 48.7         296: 77.8 / 36.2 / 48.9    340: 96.1 / 53.5 / 54.3
//   forward, bf16              60 heads 4.7 / 5.1 / 6.3 (T = 16), 3.7 / 3.7 / 4.3 (T = 8), 3.4 / 3.1 / 3.3 (T = 4)
//                             256: 14.2 / 7.6 / 8.2 (T = 16), 10.2 / 5.5 / 5.4 (T = 8), 9.4 / 4.5 / 4.2 (T = 4), 7.0 / 3.7 / 3.1 (T = 1)
//   backward, 128 tokens fp32  10 heads 26.2 / 30.1 / 34.6     12: 31.3 / 29.9 / 34.6     60: 75.9 / 45.7 / 65.3
//                             148: 147 / 79.1 / 87.1          296: 289 / 123 / 125       340: 334 / 159 / 134
// so NC = 1 up to half a head per SM forward and a fourteenth backward (three roles, and both rows and columns of the
// state to read), NC = 2 up to two heads per SM, but not for calls so short that the state is most of the work.
enum { SHAPE_1, SHAPE_2, SHAPE_4 };
int pick_shape(const wkv_args_t *a, bool backward) {
    const long long heads = (long long)a->B * a->H, sms = device_sm_count();
    if (heads * (backward ? 14 : 2) <= sms) return SHAPE_1;
    return heads <= 2 * sms && (backward || a->T >= 12) ? SHAPE_2 : SHAPE_4;
}

template <typename F, int WSRC>
int launch_fwd(const wkv_args_t *a, bool floor, cudaStream_t s) {
    SerialParams P = make_params(a);
    P.floor = floor;
    const int bh = a->B * a->H;
    switch (pick_shape(a, false)) {
        case SHAPE_1: return launch_chained(k_serial_fwd<F, WSRC, 1, 1>, dim3(bh * 8), dim3(64), 0, s, P);
        case SHAPE_2: return launch_chained(k_serial_fwd<F, WSRC, 2, 2>, dim3(bh * 2), dim3(96), 0, s, P);
        default: return launch_chained(k_serial_fwd<F, WSRC, 4, 2>, dim3(bh), dim3(96), 0, s, P);
    }
}

template <typename F, int WSRC>
int launch_bwd(const wkv_args_t *a, cudaStream_t s) {
    if (a->T == 0) {      // nothing but the state gradient to hand on
        const size_t row = (size_t)a->B * a->H * N * sizeof(float);
        cudaError_t e = cudaMemsetAsync(a->gu, 0, row, s);
        if (e == cudaSuccess && WSRC == W_STATIC) e = cudaMemsetAsync(a->gw, 0, row, s);
        if (e == cudaSuccess && a->gstate_in)
            e = a->gstate_out ? cudaMemcpyAsync(a->gstate_in, a->gstate_out, row * N, cudaMemcpyDeviceToDevice, s)
                              : cudaMemsetAsync(a->gstate_in, 0, row * N, s);
        return e == cudaSuccess ? WKV_OK : WKV_ERR_LAUNCH;
    }
    SerialParams P = make_params(a);
    const size_t n = (size_t)a->B * a->T * a->H * N;
    P.q = (float *)a->workspace; P.p = P.q + n; P.eT = P.p + n;
    const int bh = a->B * a->H;
    int err;
    switch (pick_shape(a, true)) {
        case SHAPE_1: err = launch_chained(k_serial_bwd<F, WSRC, 1, 1>, dim3(bh * 8, 3), dim3(64), 0, s, P); break;
        case SHAPE_2: err = launch_chained(k_serial_bwd<F, WSRC, 2, 2>, dim3(bh * 2, 3), dim3(96), 0, s, P); break;
        default: err = launch_chained(k_serial_bwd<F, WSRC, 4, 2>, dim3(bh, 3), dim3(96), 0, s, P);
    }
    if (err != WKV_OK) return err;
    return launch_chained(k_serial_gw<F, WSRC>, dim3(bh), dim3(1024), 0, s, P, a->gw);
}

template <typename F>
int forward_as(const wkv_args_t *a, bool pt, bool floor, cudaStream_t s) {
    if (!pt) return launch_fwd<F, W_STATIC>(a, floor, s);
    return a->w_kind == WKV_W_RAW ? launch_fwd<F, W_X>(a, floor, s) : launch_fwd<F, W_EW>(a, floor, s);
}
template <typename F>
int backward_as(const wkv_args_t *a, bool pt, cudaStream_t s) {
    if (!pt) return launch_bwd<F, W_STATIC>(a, s);
    return a->w_kind == WKV_W_RAW ? launch_bwd<F, W_X>(a, s) : launch_bwd<F, W_EW>(a, s);
}

}  // namespace

size_t scalar_backward_workspace(const wkv_args_t *a) {
    return ((size_t)a->B * a->T * 2 + a->B) * a->H * a->N * sizeof(float);
}

int scalar_forward(const wkv_args_t *a, bool pt, bool floor, cudaStream_t s) {
    switch (a->dtype) {
        case WKV_F32: return forward_as<float>(a, pt, floor, s);
        case WKV_BF16: return forward_as<__nv_bfloat16>(a, pt, floor, s);
        case WKV_F16: return forward_as<__half>(a, pt, floor, s);
    }
    return WKV_ERR_DTYPE;
}

int scalar_backward(const wkv_args_t *a, bool pt, cudaStream_t s) {
    switch (a->dtype) {
        case WKV_F32: return backward_as<float>(a, pt, s);
        case WKV_BF16: return backward_as<__nv_bfloat16>(a, pt, s);
        case WKV_F16: return backward_as<__half>(a, pt, s);
    }
    return WKV_ERR_DTYPE;
}

}  // namespace wkv
