// v4 WKV, parallel over time: one kernel forward, one backward, every tensor read once.
//
// One thread per (batch, channel) chain leaves a B200 mostly idle and waits for every token.  The state
// recurrence is linear in (p, q) with a constant decay per token, so pieces of the token axis can be
// summarised independently and folded:  a (earlier) then b of n tokens:
//   o' = o_a + n w;  m = max(o', o_b);  (p,q) = e^{o'-m}(p_a,q_a) + e^{o_b-m}(p_b,q_b);  o = m
// -- the max-shift the serial kernel makes token by token.  The state gradient (gp,gq,go) folds the same
// way in reverse.
//
// A CTA owns 16 channels of one batch row and walks the tokens in slabs of 8*NT; thread = one channel, one
// tile of 8 tokens.  Per slab:
//   forward   every thread summarises its tile from an empty state; the NT summaries meet in shared memory;
//             every thread folds those before it onto the carried state and runs its tile from there -> y.
//   backward  slabs in reverse.  Every thread recomputes y, 1/denominator and the exponent of its 8 tokens from the
//             state at its tile's start, runs the reverse recurrence over them from an empty gradient, folds the
//             summaries of the tiles after it onto the carried gradient and runs them again -> gk, gv.
// The tile's tokens stay on chip between the two sweeps (in shared memory, filled by cp.async a slab ahead), so
// k, v, gy cross HBM once: 12 + 20 bytes per token and channel in fp32, plus what forward leaves for backward:
// the state at the start of every tile (3 floats per 8 tokens).  gw needs no running derivative across
// tiles: with the true gradient at its own tile's end a tile's contribution is complete.
//
// The CTAs (B * C/16 of them) are all resident at once at the sizes that matter (8 CTAs of 128 threads and
// 64 registers per SM), so nothing waits for a second wave; with few of them the slab is made longer (NT 16, 32)
// and the walk shorter.  What bounds it: instruction issue (about 45 instructions per token-channel forward, 90
// backward) and HBM in the same range; bf16 by issue alone.
//
// Exponents are carried in base 2 inside the kernels (ex2 needs no multiply then) and converted at the
// boundaries.  Per-tile arithmetic is the math of RWKV-v4neo/cuda/wkv_cuda_bf16.cu:7-158.
#include "wkv4_common.cuh"

namespace wkv {
namespace {

constexpr int CT = 16;      // channels per CTA
constexpr int TK = 8;       // tokens per tile (one thread)
constexpr int COARSE = 64;  // tokens between the states kept when forward left nothing

struct St {
    float p, q, o;
};
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// (A,E) = (2^{a-m}, 2^{b-m}), m = max(a,b): one ex2
__device__ __forceinline__ void exp2_pair(float a, float b, float &A, float &E, float &m) {
    const float d = a - b, e = ex2(-fabsf(d));
    const bool ge = d >= 0.f;
    A = ge ? 1.f : e;
    E = ge ? e : 1.f;
    m = fmaxf(a, b);
}
// `a`, then `nw` of decay, then `b`
__device__ __forceinline__ St fold(const St &a, float nw, const St &b) {
    float A, E, m;
    exp2_pair(a.o + nw, b.o, A, E, m);
    return St{fmaf(A, a.p, E * b.p), fmaf(A, a.q, E * b.q), m};
}

struct Par {
    int B, T, C, nslab;
    Decay4 w;
    const void *u, *k, *v, *gy;
    const float *state_in, *gstate_out;
    void *y, *gk, *gv;
    float *state_out, *gstate_in, *gw, *gu;
    float *fine;        // [B][T/8][3][C]: state at the start of every tile (exponent in base 2), or NULL
    float *coarse;      // [B][T/64][3][C]: at the start of every 64 tokens, or NULL
};

// Shared memory: the slab's k, v (and gy) as [stage][tensor][tile][8 tokens + 1 of padding][16 channels] -- the
// padding keeps the two tiles a warp reads in different banks -- then the tile summaries.
template <typename F, int NT, int NTENS, bool ASYNC> struct Smem {
    static constexpr int TILE = (TK + 1) * CT;                  // elements
    F slab[ASYNC ? 2 : 1][NTENS][ASYNC ? NT * TILE : 1];
    St sum[NT][CT];
    St gsum[NT / 8][CT];
    St carry[2][CT];
};

// Copy slab `s` of the tensors to shared memory, 16 bytes at a time.  Rows past the end and channels past the last
// are zero-filled.
template <typename F, int NT, int NTENS, class S>
__device__ __forceinline__ void fetch_slab(S &sm, int stage, const F *const (&src)[NTENS], int T, int C, int c0, int t0, int tid) {
    constexpr int PER = 16 / sizeof(F), CPR = CT / PER;         // elements per chunk, chunks per row
#pragma unroll
    for (int n = 0; n < NTENS; n++)
#pragma unroll
        for (int i = 0; i < (NT * TK * CPR) / (NT * CT); i++) {
            const int x = tid + i * NT * CT, row = x / CPR, ch = (x % CPR) * PER, t = t0 + row;
            const bool in = t < T && c0 + ch < C;
            const F *g = in ? src[n] + (size_t)t * C + c0 + ch : src[n];
            const uint32_t d = (uint32_t)__cvta_generic_to_shared(
                &sm.slab[stage][n][(row / TK) * S::TILE + (row % TK) * CT + ch]);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(g), "r"(in ? 16 : 0) : "memory");
        }
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_wait0() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// What thread (tile i, channel c) starts from: `carry` folded with everything between the slab's edge and tile i --
// the tiles before i, or (REV) the tiles after it.  `mine` is this tile's summary, len(j) the tokens of tile j.
// The tile at the far edge leaves the next slab's carry in `next`.  Contains the barriers.
template <int NT, bool REV, class S, class Len>
__device__ __forceinline__ St fold_tiles(S &sm, const St &mine, const St &carry, int i, int c, float w, Len len, St *next) {
    sm.sum[i][c] = mine;
    __syncthreads();
    const int g = i >> 3, k = REV ? 7 - (i & 7) : (i & 7);      // group of eight tiles; how many of it are in between
    auto at = [&](int j) { return REV ? 8 * g + 7 - j : 8 * g + j; };
    St s = NT == 8 ? carry : St{0.f, 0.f, V4_MIN_VALUE};
    int n = 0;
    for (int j = 0; j < k; j++) {
        const int l = len(at(j));
        s = fold(s, (float)l * w, sm.sum[at(j)][c]);
        n += l;
    }
    if constexpr (NT > 8) {
        if (k == 7) sm.gsum[g][c] = fold(s, (float)len(i) * w, mine);
        __syncthreads();
        St t = carry;
        for (int j = REV ? NT / 8 - 1 : 0; REV ? j > g : j < g; j += REV ? -1 : 1) {
            int l = 0;
#pragma unroll
            for (int e = 0; e < 8; e++) l += len(8 * j + e);
            t = fold(t, (float)l * w, sm.gsum[j][c]);
        }
        s = fold(t, (float)n * w, s);
    }
    if (i == (REV ? 0 : NT - 1)) *next = fold(s, (float)len(i) * w, mine);
    return s;
}

// ---------------------------------------------------------------------------------------------- forward
// STATES: only the coarse states are wanted (backward without a hand-over)
template <typename F, int NT, bool ASYNC, bool STATES>
__global__ void __launch_bounds__(NT * CT, NT == 8 ? 8 : NT == 16 ? 4 : 2) k_v4_par_fwd(const Par P) {
    pdl_wait();
    pdl_trigger();
    typedef Smem<F, NT, 2, ASYNC> S;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    S &sm = *reinterpret_cast<S *>(smem_raw);
    const int ncb = (P.C + CT - 1) / CT, b = blockIdx.x / ncb, c0 = (blockIdx.x - b * ncb) * CT;
    const int tid = threadIdx.x, c = tid & (CT - 1), i = tid / CT, ch = min(c0 + c, P.C - 1), T = P.T, C = P.C;
    const bool live = c0 + c < C;
    const float w = P.w.at(ch) * V4_LOG2E, u = Elem<F>::ld((const F *)P.u + ch) * V4_LOG2E;
    const size_t row = (size_t)b * T * C, so = ((size_t)b * C + ch) * 3;
    const F *const src[2] = {(const F *)P.k + row, (const F *)P.v + row};
    if (i == 0)
        sm.carry[0][c] = P.state_in ? St{P.state_in[so], P.state_in[so + 1], to_base2(P.state_in[so + 2])} : St{0.f, 0.f, V4_MIN_VALUE};
    if (ASYNC) { fetch_slab<F, NT, 2>(sm, 0, src, T, C, c0, 0, tid); cp_commit(); }
    const int n8 = (T + TK - 1) / TK, n64 = (T + COARSE - 1) / COARSE;

    for (int s = 0; s < P.nslab; s++) {
        const int t0 = s * NT * TK, mine0 = t0 + i * TK;      // first token of the slab, of this tile
        if (ASYNC) cp_wait0();
        __syncthreads();
        if (ASYNC && s + 1 < P.nslab) { fetch_slab<F, NT, 2>(sm, (s + 1) & 1, src, T, C, c0, t0 + NT * TK, tid); cp_commit(); }
        auto len = [&](int j) { return min(TK, max(0, T - t0 - j * TK)); };
        const int n = len(i);
        float kk[TK], vv[TK];
#pragma unroll
        for (int j = 0; j < TK; j++) {
            if (ASYNC) {
                kk[j] = Elem<F>::ld(&sm.slab[s & 1][0][i * S::TILE + j * CT + c]) * V4_LOG2E;
                vv[j] = Elem<F>::ld(&sm.slab[s & 1][1][i * S::TILE + j * CT + c]);
            } else {
                const size_t o = (size_t)min(mine0 + j, T - 1) * C + ch;
                kk[j] = Elem<F>::ld(src[0] + o) * V4_LOG2E;
                vv[j] = Elem<F>::ld(src[1] + o);
            }
        }
        St a{0.f, 0.f, V4_MIN_VALUE};
#pragma unroll
        for (int j = 0; j < TK; j++)
            if (j < n) {
                float A, E, m;
                exp2_pair(w + a.o, kk[j], A, E, m);
                a.p = fmaf(A, a.p, E * vv[j]); a.q = fmaf(A, a.q, E); a.o = m;
            }
        St x = fold_tiles<NT, false>(sm, a, sm.carry[s & 1][c], i, c, w, len, &sm.carry[(s + 1) & 1][c]);
        if (live && n > 0) {
            if (!STATES && P.fine) {
                float *f = P.fine + ((size_t)b * n8 + mine0 / TK) * 3 * C + ch;
                f[0] = x.p; f[C] = x.q; f[2 * (size_t)C] = x.o;
            }
            if (P.coarse && (i & 7) == 0) {
                float *f = P.coarse + ((size_t)b * n64 + mine0 / COARSE) * 3 * C + ch;
                f[0] = x.p; f[C] = x.q; f[2 * (size_t)C] = x.o;
            }
        }
        if (!STATES) {
            F *y = (F *)P.y + row + ch;
#pragma unroll
            for (int j = 0; j < TK; j++)
                if (j < n) {
                    float A, E, m;
                    exp2_pair(x.o, u + kk[j], A, E, m);
                    const float out = __fdividef(fmaf(A, x.p, E * vv[j]), fmaf(A, x.q, E));
                    if (live) Elem<F>::st(y + (size_t)(mine0 + j) * C, out);
                    exp2_pair(w + x.o, kk[j], A, E, m);
                    x.p = fmaf(A, x.p, E * vv[j]); x.q = fmaf(A, x.q, E); x.o = m;
                }
        }
    }
    if (!STATES && P.state_out) {
        __syncthreads();
        if (i == 0 && live) {
            const St f = sm.carry[P.nslab & 1][c];
            P.state_out[so] = f.p; P.state_out[so + 1] = f.q; P.state_out[so + 2] = from_base2(f.o);
        }
    }
}

// ---------------------------------------------------------------------------------------------- backward
// FINE: forward left the state at the start of every tile; else the slab's states are rebuilt from the coarse ones
// (or, one slab only, from state_in) by one more summary and fold.
template <typename F, int NT, bool ASYNC, bool FINE>
__global__ void __launch_bounds__(NT * CT, NT == 8 ? 7 : NT == 16 ? 3 : 1) k_v4_par_bwd(const Par P) {
    pdl_wait();
    pdl_trigger();
    typedef Smem<F, NT, 3, ASYNC> S;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    S &sm = *reinterpret_cast<S *>(smem_raw);
    const int ncb = (P.C + CT - 1) / CT, b = blockIdx.x / ncb, c0 = (blockIdx.x - b * ncb) * CT;
    const int tid = threadIdx.x, c = tid & (CT - 1), i = tid / CT, ch = min(c0 + c, P.C - 1), T = P.T, C = P.C;
    const bool live = c0 + c < C;
    const float wn = P.w.at(ch), w = wn * V4_LOG2E, u = Elem<F>::ld((const F *)P.u + ch) * V4_LOG2E;
    const size_t row = (size_t)b * T * C, so = ((size_t)b * C + ch) * 3;
    const F *const src[3] = {(const F *)P.k + row, (const F *)P.v + row, (const F *)P.gy + row};
    const int n8 = (T + TK - 1) / TK, n64 = (T + COARSE - 1) / COARSE, last = P.nslab - 1;
    if (i == 0) {
        St g{0.f, 0.f, V4_MIN_VALUE};
        if (P.gstate_out) {
            g.p = P.gstate_out[so]; g.q = P.gstate_out[so + 1];
            if (g.p != 0.f || g.q != 0.f) g.o = to_base2(P.gstate_out[so + 2]);
        }
        sm.carry[last & 1][c] = g;
    }
    // the state at the start of this thread's tile (FINE) or of the 64 tokens around it, for slab s
    auto start_state = [&](int s) {
        const int t = s * NT * TK + i * TK;
        if (!FINE && !P.coarse) return P.state_in ? St{P.state_in[so], P.state_in[so + 1], to_base2(P.state_in[so + 2])} : St{0.f, 0.f, V4_MIN_VALUE};
        const float *f = FINE ? P.fine + ((size_t)b * n8 + min(t / TK, n8 - 1)) * 3 * C + ch
                              : P.coarse + ((size_t)b * n64 + min(t / COARSE, n64 - 1)) * 3 * C + ch;
        return St{f[0], f[C], f[2 * (size_t)C]};
    };
    St x = start_state(last);
    if (ASYNC) { fetch_slab<F, NT, 3>(sm, last & 1, src, T, C, c0, last * NT * TK, tid); cp_commit(); }
    float gw = 0.f, gu = 0.f;

    for (int s = last; s >= 0; s--) {
        const int t0 = s * NT * TK, mine0 = t0 + i * TK;
        if (ASYNC) cp_wait0();
        __syncthreads();
        St x_next;
        if (s > 0) {
            if (ASYNC) { fetch_slab<F, NT, 3>(sm, (s - 1) & 1, src, T, C, c0, t0 - NT * TK, tid); cp_commit(); }
            x_next = start_state(s - 1);
        }
        auto len = [&](int j) { return min(TK, max(0, T - t0 - j * TK)); };
        const int n = len(i);
        auto ld = [&](int tens, int j) {
            return Elem<F>::ld(ASYNC ? &sm.slab[s & 1][tens][i * S::TILE + j * CT + c] : src[tens] + (size_t)min(mine0 + j, T - 1) * C + ch);
        };
        if constexpr (!FINE) {
            // the state at the tile's start: fold the summaries of the tiles between the kept state and it.
            // Without `coarse` there is one slab and the kept state is the initial one.
            St a{0.f, 0.f, V4_MIN_VALUE};
#pragma unroll
            for (int j = 0; j < TK; j++)
                if (j < n) {
                    float A, E, m;
                    const float k = ld(0, j) * V4_LOG2E, v = ld(1, j);
                    exp2_pair(w + a.o, k, A, E, m);
                    a.p = fmaf(A, a.p, E * v); a.q = fmaf(A, a.q, E); a.o = m;
                }
            sm.sum[i][c] = a;
            __syncthreads();
            for (int j = P.coarse ? (i & ~7) : 0; j < i; j++) x = fold(x, (float)len(j) * w, sm.sum[j][c]);
            __syncthreads();
        }
        float ys[TK], zs[TK], ze[TK];      // y, gy / denominator, exponent of the token's own term in it
        float dpdw = 0.f, dqdw = 0.f;      // d(p,q)/dw since the tile's start
#pragma unroll
        for (int j = 0; j < TK; j++)
            if (j < n) {
                float A, E, m;
                const float k = ld(0, j) * V4_LOG2E, v = ld(1, j), g = ld(2, j);
                exp2_pair(x.o, u + k, A, E, m);
                const float iden = __fdividef(1.f, fmaf(A, x.q, E));
                ys[j] = fmaf(A, x.p, E * v) * iden;
                zs[j] = g * iden;
                ze[j] = k + u - m;
                gw = fmaf(zs[j] * A, fmaf(-dqdw, ys[j], dpdw), gw);
                gu = fmaf(zs[j] * E, v - ys[j], gu);
                exp2_pair(w + x.o, k, A, E, m);
                dpdw = A * (x.p + dpdw); dqdw = A * (x.q + dqdw);
                x.p = fmaf(A, x.p, E * v); x.q = fmaf(A, x.q, E); x.o = m;
            }
        // reverse over the tile from an empty gradient
        St a{0.f, 0.f, V4_MIN_VALUE};
#pragma unroll
        for (int j = TK - 1; j >= 0; j--)
            if (j < n) {
                float A, E, m;
                exp2_pair(w + a.o, ze[j] - ld(0, j) * V4_LOG2E - u, A, E, m);
                E *= zs[j];
                a.p = fmaf(A, a.p, E); a.q = fmaf(A, a.q, -E * ys[j]); a.o = m;
            }
        St g = fold_tiles<NT, true>(sm, a, sm.carry[s & 1][c], i, c, w, len, &sm.carry[(s + 1) & 1][c]);
        // what the gradient at the tile's end sees of the decay inside the tile
        if (n > 0) gw = fmaf(fmaf(g.p, dpdw, g.q * dqdw), ex2(x.o + g.o), gw);
        F *gk = (F *)P.gk + row + ch, *gv = (F *)P.gv + row + ch;
#pragma unroll
        for (int j = TK - 1; j >= 0; j--)
            if (j < n) {
                const float k = ld(0, j) * V4_LOG2E, v = ld(1, j);
                float A = zs[j] * ex2(ze[j]), E = ex2(k + g.o), m;
                if (live) {
                    Elem<F>::st(gk + (size_t)(mine0 + j) * C, fmaf(A, v - ys[j], E * fmaf(g.p, v, g.q)));
                    Elem<F>::st(gv + (size_t)(mine0 + j) * C, fmaf(E, g.p, A));
                }
                exp2_pair(w + g.o, ze[j] - k - u, A, E, m);
                E *= zs[j];
                g.p = fmaf(A, g.p, E); g.q = fmaf(A, g.q, -E * ys[j]); g.o = m;
            }
        x = x_next;
    }
    // the tiles' shares of gw and gu, summed in a fixed order
    __syncthreads();
    sm.sum[i][c] = St{gw, gu, 0.f};
    __syncthreads();
    if (i == 0 && live) {
        float a = 0.f, e = 0.f;
#pragma unroll 8
        for (int j = 0; j < NT; j++) { a += sm.sum[j][c].p; e += sm.sum[j][c].q; }
        P.gw[(size_t)b * C + ch] = a * wn;
        P.gu[(size_t)b * C + ch] = e;
        if (P.gstate_in) {
            const St f = sm.carry[1][c];      // (slab 0 leaves its carry there)
            P.gstate_in[so] = f.p; P.gstate_in[so + 1] = f.q; P.gstate_in[so + 2] = from_base2(f.o);
        }
    }
}

// Tiles per slab: 8 (8 CTAs of 128 threads per SM) once the CTAs alone fill the SMs; else longer slabs, and never
// much longer than the segment.
int pick_tiles(int B, int T, int C) {
    const long long ctas = (long long)B * ((C + CT - 1) / CT), sms = device_sm_count();
    if (ctas >= 4 * sms || T <= 64) return 8;
    return ctas >= 2 * sms || T <= 128 ? 16 : 32;
}

template <class K>
int launch(K kern, size_t smem, unsigned char (&attr_done)[64], const Par &P, int nt, cudaStream_t s) {
    if (!set_max_smem_once(kern, (int)smem, attr_done)) return WKV_ERR_LAUNCH;
    return launch_chained(kern, dim3(P.B * ((P.C + CT - 1) / CT)), dim3(nt * CT), smem, s, P);
}
template <typename F, int NT, bool ASYNC>
int launch_fwd(Par P, bool states, cudaStream_t s) {
    static unsigned char done[2][64];
    P.nslab = (P.T + NT * TK - 1) / (NT * TK);
    const size_t smem = sizeof(Smem<F, NT, 2, ASYNC>);
    return states ? launch(k_v4_par_fwd<F, NT, ASYNC, true>, smem, done[0], P, NT, s)
                  : launch(k_v4_par_fwd<F, NT, ASYNC, false>, smem, done[1], P, NT, s);
}
template <typename F, int NT, bool ASYNC>
int launch_bwd(Par P, cudaStream_t s) {
    static unsigned char done[2][64];
    P.nslab = (P.T + NT * TK - 1) / (NT * TK);
    const size_t smem = sizeof(Smem<F, NT, 3, ASYNC>);
    return P.fine ? launch(k_v4_par_bwd<F, NT, ASYNC, true>, smem, done[0], P, NT, s)
                  : launch(k_v4_par_bwd<F, NT, ASYNC, false>, smem, done[1], P, NT, s);
}

// 16-byte copies need rows that start on 16 bytes; other widths load element by element
template <typename F>
bool rows_aligned(const Par &P) {
    return (size_t)P.C * sizeof(F) % 16 == 0 && aligned16(P.k) && aligned16(P.v) && (!P.gy || aligned16(P.gy));
}

template <typename F>
int forward_as(const Par &P, bool states, cudaStream_t s) {
    if (!rows_aligned<F>(P)) return launch_fwd<F, 16, false>(P, states, s);
    switch (pick_tiles(P.B, P.T, P.C)) {
        case 8: return launch_fwd<F, 8, true>(P, states, s);
        case 16: return launch_fwd<F, 16, true>(P, states, s);
        default: return launch_fwd<F, 32, true>(P, states, s);
    }
}
template <typename F>
int backward_as(Par P, float *scratch, cudaStream_t s) {
    const bool aligned = rows_aligned<F>(P);
    const int nt = aligned ? pick_tiles(P.B, P.T, P.C) : 16;
    if (!P.fine && P.T > nt * TK) {
        // nothing was handed over and there is more than one slab: the states every 64 tokens first
        P.coarse = scratch;
        const int err = forward_as<F>(P, true, s);
        if (err != WKV_OK) return err;
    }
    if (!aligned) return launch_bwd<F, 16, false>(P, s);
    switch (nt) {
        case 8: return launch_bwd<F, 8, true>(P, s);
        case 16: return launch_bwd<F, 16, true>(P, s);
        default: return launch_bwd<F, 32, true>(P, s);
    }
}

Par make_par(int B, int T, int C, const Decay4 &w, const void *u, const void *k, const void *v, const float *si) {
    Par P = {};
    P.B = B; P.T = T; P.C = C; P.w = w; P.u = u; P.k = k; P.v = v; P.state_in = si;
    return P;
}

}  // namespace

size_t v4_par_ckpt_bytes(int B, int T, int C) { return (size_t)B * ((T + TK - 1) / TK) * 3 * C * sizeof(float); }

int v4_par_forward(int B, int T, int C, int dtype, const Decay4 &w, const void *u, const void *k, const void *v,
                   const float *si, void *y, float *so, float *ckpt, cudaStream_t s) {
    Par P = make_par(B, T, C, w, u, k, v, si);
    P.y = y; P.state_out = so; P.fine = ckpt;
    switch (dtype) {
        case WKV_F32: return forward_as<float>(P, false, s);
        case WKV_BF16: return forward_as<__nv_bfloat16>(P, false, s);
        case WKV_F16: return forward_as<__half>(P, false, s);
    }
    return WKV_ERR_DTYPE;
}

int v4_par_backward(int B, int T, int C, int dtype, const Decay4 &w, const void *u, const void *k, const void *v,
                    const float *si, const void *gy, const float *gso, float *gw, float *gu, void *gk, void *gv,
                    float *gsi, float *ws, const float *ckpt, cudaStream_t s) {
    Par P = make_par(B, T, C, w, u, k, v, si);
    P.gy = gy; P.gstate_out = gso; P.gw = gw; P.gu = gu; P.gk = gk; P.gv = gv; P.gstate_in = gsi;
    P.fine = const_cast<float *>(ckpt);
    switch (dtype) {
        case WKV_F32: return backward_as<float>(P, ws, s);
        case WKV_BF16: return backward_as<__nv_bfloat16>(P, ws, s);
        case WKV_F16: return backward_as<__half>(P, ws, s);
    }
    return WKV_ERR_DTYPE;
}

}  // namespace wkv
