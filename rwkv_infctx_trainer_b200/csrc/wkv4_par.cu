// v4 WKV, parallel over time: one kernel forward, one backward, every tensor read once.
//
// One thread per (batch, channel) chain leaves a B200 mostly idle and waits for every token.  The state
// recurrence is linear in (p, q) with a constant decay per token, so pieces of the token axis can be
// summarised independently and folded:  a (earlier) then b of n tokens:
//   o' = o_a + n w;  m = max(o', o_b);  (p,q) = e^{o'-m}(p_a,q_a) + e^{o_b-m}(p_b,q_b);  o = m
// -- the max-shift the serial kernel makes token by token.  The state gradient (gp,gq,go) folds the same
// way in reverse.
//
// A CTA owns 16 channels of one batch row and walks the tokens in slabs of 8*NT; thread = two adjacent
// channels, one tile of 8 tokens.  Per slab:
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
// The slab is as long as leaves the CTAs (B * C/16 of them) all resident at once (see pick_tiles), so that nothing waits for a
// second wave and the walk is short.
// Issue slots and HBM time are of the same size here, so the inner loops work on channel pairs: the packed fp32
// instructions (fma.f32x2) take two channels each, and so does every address, load and store.
//
// Exponents are carried in base 2 inside the kernels (ex2 needs no multiply then) and converted at the
// boundaries.
//
// Inside a tile the max-shift is done once.  With one reference exponent M for the tile's 8 tokens, p~ = p 2^{o-M}
// and e_t = 2^{k_t-M}, a token is  y = (p~ + U e v) / (q~ + U e),  p~ <- W p~ + e v,  q~ <- W q~ + e  with W = e^w and U = e^u
// constant: one ex2 and one reciprocal instead of two max-shifted pairs, and the reverse recurrence needs no exponential at
// all (gp <- W gp + z, gq <- W gq - z y with z = gy / denominator).  That is sound while nothing leaves the fp32
// range: |u| plus the distance of any k from M at most 60, the incoming state at most 2^60 above M, the incoming
// gradient at most 2^90.  A CTA that meets a tile that is not tame in this sense starts its walk over by the
// token-by-token max-shift of RWKV-v4neo/cuda/wkv_cuda_bf16.cu:7-158; both keep the same state representation (o =
// the running maximum) at tile boundaries.
#include <type_traits>

#include "wkv4_common.cuh"

namespace wkv {
namespace {

constexpr int CT = 16;      // channels per CTA
constexpr int CP = CT / 2;  // threads (channel pairs) per tile
constexpr int TK = 8;       // tokens per tile (one thread)
constexpr int COARSE = 64;  // tokens between the states kept when forward left nothing
constexpr float RANGE = 60.f;        // how far (log2) a tame tile's exponents may lie from its reference
constexpr float GRAD_RANGE = 90.f;

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// ---- two channels at a time
// keeps loads of later tokens from being hoisted above this point: all eight at once do not fit the registers
__device__ __forceinline__ void no_hoist() { asm volatile("" ::: "memory"); }
__device__ __forceinline__ f2 max2(f2 a, f2 b) { return make_float2(fmaxf(a.x, b.x), fmaxf(a.y, b.y)); }
__device__ __forceinline__ f2 min2(f2 a, f2 b) { return make_float2(fminf(a.x, b.x), fminf(a.y, b.y)); }
__device__ __forceinline__ f2 ex2_2(f2 a) { return make_float2(ex2(a.x), ex2(a.y)); }
__device__ __forceinline__ f2 rcp2(f2 a) { return make_float2(rcp(a.x), rcp(a.y)); }
struct St {
    f2 p, q, o;
};
__device__ __forceinline__ St empty_state() { return St{both(0.f), both(0.f), both(V4_MIN_VALUE)}; }
// `a`, then `nw` of decay, then `b`
__device__ __forceinline__ St fold(const St &a, f2 nw, const St &b) {
    const f2 d = add2(a.o, nw), m = max2(d, b.o), A = ex2_2(sub2(d, m)), E = ex2_2(sub2(b.o, m));
    return St{fma2(A, a.p, mul2(E, b.p)), fma2(A, a.q, mul2(E, b.q)), m};
}

// ---- two adjacent elements
template <typename F> struct Pair;
template <> struct Pair<float> {
    static __device__ __forceinline__ f2 ld(const float *p) { return *reinterpret_cast<const f2 *>(p); }
    static __device__ __forceinline__ void st(float *p, f2 v) { *reinterpret_cast<f2 *>(p) = v; }
};
template <> struct Pair<__nv_bfloat16> {
    static __device__ __forceinline__ f2 ld(const __nv_bfloat16 *p) {
        return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(p));
    }
    static __device__ __forceinline__ void st(__nv_bfloat16 *p, f2 v) { *reinterpret_cast<__nv_bfloat162 *>(p) = __floats2bfloat162_rn(v.x, v.y); }
};
template <> struct Pair<__half> {
    static __device__ __forceinline__ f2 ld(const __half *p) { return __half22float2(*reinterpret_cast<const __half2 *>(p)); }
    static __device__ __forceinline__ void st(__half *p, f2 v) { *reinterpret_cast<__half2 *>(p) = __floats2half2_rn(v.x, v.y); }
};

// ---- One tile, one channel, by the token-by-token max-shift: what a CTA falls back to.
// (A,E) = (2^{a-m}, 2^{b-m}), m = max(a,b): one ex2
__device__ __forceinline__ void exp2_pair(float a, float b, float &A, float &E, float &m) {
    const float d = a - b, e = ex2(-fabsf(d));
    const bool ge = d >= 0.f;
    A = ge ? 1.f : e;
    E = ge ? e : 1.f;
    m = fmaxf(a, b);
}
struct Slow {
    float p, q, o;
};
// token j of the tile: element j * stride of k, v, gy
template <typename F>
__device__ __noinline__ Slow slow_summary(const F *k, const F *v, size_t stride, int n, float w) {
    Slow a{0.f, 0.f, V4_MIN_VALUE};
    for (int j = 0; j < n; j++) {
        float A, E, m;
        exp2_pair(w + a.o, Elem<F>::ld(k + j * stride) * V4_LOG2E, A, E, m);
        a.p = fmaf(A, a.p, E * Elem<F>::ld(v + j * stride)); a.q = fmaf(A, a.q, E); a.o = m;
    }
    return a;
}
template <typename F>
__device__ __noinline__ void slow_apply(const F *k, const F *v, size_t stride, int n, float w, float u, Slow x, F *y, size_t C) {
    for (int j = 0; j < n; j++) {
        float A, E, m;
        const float kj = Elem<F>::ld(k + j * stride) * V4_LOG2E, vj = Elem<F>::ld(v + j * stride);
        exp2_pair(x.o, u + kj, A, E, m);
        Elem<F>::st(y + j * C, __fdividef(fmaf(A, x.p, E * vj), fmaf(A, x.q, E)));
        exp2_pair(w + x.o, kj, A, E, m);
        x.p = fmaf(A, x.p, E * vj); x.q = fmaf(A, x.q, E); x.o = m;
    }
}
struct SlowGrads {
    Slow a;                             // the reverse summary from an empty gradient
    float gw, gu, dpdw, dqdw, o_end;
};
// x: the state at the tile's start.  With gk given, also the outputs, from the gradient g at the tile's end.
template <typename F>
__device__ __noinline__ SlowGrads slow_backward(const F *k, const F *v, const F *gy, size_t stride, int n, float w, float u, Slow x,
                                                Slow g, F *gk, F *gv, size_t C) {
    float ys[TK], zs[TK], ze[TK];
    SlowGrads r{};
    for (int j = 0; j < n; j++) {
        float A, E, m;
        const float kj = Elem<F>::ld(k + j * stride) * V4_LOG2E, vj = Elem<F>::ld(v + j * stride);
        exp2_pair(x.o, u + kj, A, E, m);
        const float iden = __fdividef(1.f, fmaf(A, x.q, E));
        ys[j] = fmaf(A, x.p, E * vj) * iden;
        zs[j] = Elem<F>::ld(gy + j * stride) * iden;
        ze[j] = kj + u - m;
        r.gw = fmaf(zs[j] * A, fmaf(-r.dqdw, ys[j], r.dpdw), r.gw);
        r.gu = fmaf(zs[j] * E, vj - ys[j], r.gu);
        exp2_pair(w + x.o, kj, A, E, m);
        r.dpdw = A * (x.p + r.dpdw); r.dqdw = A * (x.q + r.dqdw);
        x.p = fmaf(A, x.p, E * vj); x.q = fmaf(A, x.q, E); x.o = m;
    }
    r.o_end = x.o;
    for (int j = n - 1; j >= 0; j--) {
        float A, E, m;
        const float kj = Elem<F>::ld(k + j * stride) * V4_LOG2E, vj = Elem<F>::ld(v + j * stride);
        if (gk) {
            const float t = zs[j] * ex2(ze[j]), e = ex2(kj + g.o);
            Elem<F>::st(gk + j * C, fmaf(t, vj - ys[j], e * fmaf(g.p, vj, g.q)));
            Elem<F>::st(gv + j * C, fmaf(e, g.p, t));
        }
        exp2_pair(w + g.o, ze[j] - kj - u, A, E, m);
        E *= zs[j];
        g.p = fmaf(A, g.p, E); g.q = fmaf(A, g.q, -E * ys[j]); g.o = m;
    }
    r.a = g;
    return r;
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

// Shared memory: the slab's k, v (and gy) as [stage][tensor][tile][8 tokens + padding][16 channels] -- the
// padding keeps the tiles a warp reads in different banks, and in backward holds the tile's start state: 16 floats of
// p, q, o behind its k, v, gy -- then the tile summaries.
template <typename F> struct Tile {
    static constexpr int SIZE = (TK + (sizeof(F) == 4 ? 1 : 3)) * CT;   // elements
};
template <typename F, int NT, int NTENS, bool ASYNC> struct Smem {
    static constexpr int TILE = Tile<F>::SIZE;
    F slab[ASYNC ? 2 : 1][NTENS][ASYNC ? NT * TILE : 8];
    St sum[NT][CP];
    St gsum[NT / 8][CP];
    St carry[2][CP];
};

// The copies of a slab this thread makes, 16 bytes each: row r0 + i * ROWS of the slab, channels ch0 .. .
template <typename F, int NT> struct Copy {
    static constexpr int PER = 16 / sizeof(F), CPR = CT / PER;          // elements per copy, copies per row
    static constexpr int ROWS = NT * CP / CPR, N = NT * TK / ROWS;      // rows the CTA covers at once, copies per thread
    int r0, ch0;
    uint32_t dst;       // byte offset of row r0 inside a tensor's slab
    bool in;            // its channels exist
    __device__ __forceinline__ Copy(int tid, int c0, int C) {
        r0 = tid / CPR;
        ch0 = c0 + (tid % CPR) * PER;
        in = ch0 < C;
        dst = ((r0 / TK) * Tile<F>::SIZE + (r0 % TK) * CT + (tid % CPR) * PER) * sizeof(F);
    }
    static_assert(ROWS % TK == 0, "");
    static constexpr uint32_t STEP = (ROWS / TK) * Tile<F>::SIZE * sizeof(F);
};
// rows past the end and channels past the last are zero-filled
template <typename F, int NT, int NTENS, class S>
__device__ __forceinline__ void fetch_slab(S &sm, const Copy<F, NT> &cp, int stage, const F *const (&src)[NTENS], int T, int C, int t0) {
    typedef Copy<F, NT> K;
    const bool full = t0 + NT * TK <= T;
    const size_t off = (size_t)(t0 + cp.r0) * C + cp.ch0;
#pragma unroll
    for (int n = 0; n < NTENS; n++) {
        const uint32_t d = (uint32_t)__cvta_generic_to_shared(&sm.slab[stage][n][0]) + cp.dst;
#pragma unroll
        for (int i = 0; i < K::N; i++) {
            const bool in = cp.in && (full || t0 + cp.r0 + i * K::ROWS < T);
            const F *g = in ? src[n] + off + (size_t)i * K::ROWS * C : src[n];
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d + i * K::STEP), "l"(g), "r"(in ? 16 : 0) : "memory");
        }
    }
}
// The start states of the slab's tiles (rows `first` .. of [..][3][C]) to the padding of the tiles.
template <typename F, int NT, class S>
__device__ __forceinline__ void fetch_states(S &sm, int stage, const float *fine, int first, int n8, int C, int c0, int tid) {
#pragma unroll
    for (int x = tid; x < NT * 12; x += NT * CP) {
        const int tile = x / 12, r = x % 12 / 4, ch = x % 4 * 4;
        const bool in = first + tile < n8 && c0 + ch < C;
        const float *g = in ? fine + ((size_t)(first + tile) * 3 + r) * C + c0 + ch : fine;
        const uint32_t d = (uint32_t)__cvta_generic_to_shared(&sm.slab[stage][r][tile * S::TILE + TK * CT]) + ch * 4;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(g), "r"(in ? 16 : 0) : "memory");
    }
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_wait0() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// What thread (tile i, pair c) starts from: `carry` folded with everything between the slab's edge and tile i --
// the tiles before i, or (REV) the tiles after it.  `mine` is this tile's summary, len(j) the tokens of tile j.
// The tile at the far edge leaves the next slab's carry in `next`.  Contains the barriers; the first also ORs
// `bad` over the CTA, and when that is set nothing is folded and `stop` is.
template <int NT, bool REV, bool FULL, class S, class Len>
__device__ __forceinline__ St fold_tiles(S &sm, const St &mine, const St &carry, int i, int c, f2 w, Len len, St *next, bool bad, bool &stop) {
    sm.sum[i][c] = mine;
    if (__syncthreads_or(bad)) {
        stop = true;
        return carry;
    }
    const int g = i >> 3, k = REV ? 7 - (i & 7) : (i & 7);      // group of eight tiles; how many of it are in between
    auto at = [&](int j) { return REV ? 8 * g + 7 - j : 8 * g + j; };
    const f2 w8 = mul2(w, both((float)TK));
    auto decay = [&](int n) { return mul2(w, both((float)n)); };
    St s = NT == 8 ? carry : empty_state();
    int n = 0;
#pragma unroll 1
    for (int j = 0; j < k; j++) {
        const int l = FULL ? TK : len(at(j));
        s = fold(s, FULL ? w8 : decay(l), sm.sum[at(j)][c]);
        n += l;
    }
    if constexpr (NT > 8) {
        if (k == 7) sm.gsum[g][c] = fold(s, FULL ? w8 : decay(len(i)), mine);
        __syncthreads();
        St t = carry;
        for (int j = REV ? NT / 8 - 1 : 0; REV ? j > g : j < g; j += REV ? -1 : 1) {
            int l = 8 * TK;
            if (!FULL) {
                l = 0;
#pragma unroll
                for (int e = 0; e < 8; e++) l += len(8 * j + e);
            }
            t = fold(t, decay(l), sm.gsum[j][c]);
        }
        s = fold(t, decay(n), s);
    }
    if (i == (REV ? 0 : NT - 1)) *next = fold(s, FULL ? w8 : decay(len(i)), mine);
    return s;
}

// What both kernels know of their place: batch row, first channel, the pair and tile of the thread.
template <bool ASYNC> struct Place {
    int b, c0, c, i, ch, ch1, C, T;
    bool live, live1;
    size_t row;
    __device__ __forceinline__ Place(const Par &P) {
        C = P.C; T = P.T;
        const int ncb = (C + CT - 1) / CT, tid = threadIdx.x;
        b = blockIdx.x / ncb; c0 = (blockIdx.x - b * ncb) * CT;
        c = tid & (CP - 1); i = tid / CP;
        live = c0 + 2 * c < C; live1 = ASYNC ? live : c0 + 2 * c + 1 < C;
        ch = ASYNC ? (live ? c0 + 2 * c : C - 2) : min(c0 + 2 * c, C - 1);
        ch1 = ASYNC ? ch + 1 : min(ch + 1, C - 1);
        row = (size_t)b * T * C;
    }
    template <typename F> __device__ __forceinline__ f2 ld(const F *p, size_t o) const {
        if (ASYNC) return Pair<F>::ld(p + o + ch);
        return make_float2(Elem<F>::ld(p + o + ch), Elem<F>::ld(p + o + ch1));
    }
    // of a [C] vector that may start at any element
    template <typename F> __device__ __forceinline__ f2 elements(const F *p) const { return make_float2(Elem<F>::ld(p + ch), Elem<F>::ld(p + ch1)); }
    // `p` points at channel ch
    template <typename F> __device__ __forceinline__ void st(F *p, f2 v) const {
        if (ASYNC) {
            if (live) Pair<F>::st(p, v);
        } else {
            if (live) Elem<F>::st(p, v.x);
            if (live1) Elem<F>::st(p + 1, v.y);
        }
    }
    __device__ __forceinline__ St ext_state(const float *s) const {
        if (!s) return empty_state();
        const float *x = s + ((size_t)b * C + ch) * 3, *y = s + ((size_t)b * C + ch1) * 3;
        return St{make_float2(x[0], y[0]), make_float2(x[1], y[1]), make_float2(to_base2(x[2]), to_base2(y[2]))};
    }
    // (an all-zero gradient carries no exponent)
    __device__ __forceinline__ St ext_gradient(const float *s) const {
        St g = ext_state(s);
        if (g.p.x == 0.f && g.q.x == 0.f) g.o.x = V4_MIN_VALUE;
        if (g.p.y == 0.f && g.q.y == 0.f) g.o.y = V4_MIN_VALUE;
        return g;
    }
    __device__ __forceinline__ void put_state(float *s, const St &f) const {
        float *x = s + ((size_t)b * C + ch) * 3;
        if (live) { x[0] = f.p.x; x[1] = f.q.x; x[2] = from_base2(f.o.x); }
        if (live1) { x[3] = f.p.y; x[4] = f.q.y; x[5] = from_base2(f.o.y); }
    }
    // the three rows of a kept state ([..][3][C]); f points at its first row
    __device__ __forceinline__ St kept(const float *f) const { return St{ld(f, 0), ld(f, C), ld(f, 2 * (size_t)C)}; }
    __device__ __forceinline__ void keep(float *f, const St &x) const {
        st(f + ch, x.p); st(f + C + ch, x.q); st(f + 2 * (size_t)C + ch, x.o);
    }
};

// ---------------------------------------------------------------------------------------------- forward
// The whole walk by the token-by-token max-shift: a CTA that meets a tile that is not tame starts over here.
// Out of line and reached with nothing live, so that the usual path does not pay for it in registers.
template <typename F, int NT, bool ASYNC, bool STATES, class S>
__device__ __noinline__ void slow_forward(const Par &P, S &sm) {
    const Place<ASYNC> L(P);
    const int c = L.c, i = L.i, T = L.T, C = L.C, n8 = (T + TK - 1) / TK, n64 = (T + COARSE - 1) / COARSE;
    const f2 w = make_float2(P.w.at(L.ch) * V4_LOG2E, P.w.at(L.ch1) * V4_LOG2E), u = mul2(L.elements((const F *)P.u), both(V4_LOG2E));
    const F *const k = (const F *)P.k + L.row, *const v = (const F *)P.v + L.row;
    if (i == 0) sm.carry[0][c] = L.ext_state(P.state_in);
    for (int s = 0; s < P.nslab; s++) {
        __syncthreads();
        const int t0 = s * NT * TK, mine0 = t0 + i * TK;
        auto len = [&](int j) { return min(TK, max(0, T - t0 - j * TK)); };
        const int n = len(i);
        const size_t o0 = (size_t)min(mine0, T - 1) * C + L.ch, o1 = o0 - L.ch + L.ch1;
        const Slow f = slow_summary<F>(k + o0, v + o0, C, n, w.x), g = slow_summary<F>(k + o1, v + o1, C, n, w.y);
        bool stop = false;
        const St x = fold_tiles<NT, false, false>(sm, St{make_float2(f.p, g.p), make_float2(f.q, g.q), make_float2(f.o, g.o)}, sm.carry[s & 1][c], i, c, w,
                                                  len, &sm.carry[(s + 1) & 1][c], false, stop);
        if (n > 0) {
            if (!STATES && P.fine) L.keep(P.fine + ((size_t)L.b * n8 + mine0 / TK) * 3 * C, x);
            if (STATES && (i & 7) == 0) L.keep(P.coarse + ((size_t)L.b * n64 + mine0 / COARSE) * 3 * C, x);
        }
        if (!STATES) {
            F *y = (F *)P.y + L.row;
            if (L.live) slow_apply<F>(k + o0, v + o0, C, n, w.x, u.x, Slow{x.p.x, x.q.x, x.o.x}, y + o0, C);
            if (L.live1) slow_apply<F>(k + o1, v + o1, C, n, w.y, u.y, Slow{x.p.y, x.q.y, x.o.y}, y + o1, C);
        }
    }
}

// STATES: only the coarse states are wanted (backward without a hand-over)
template <typename F, int NT, bool ASYNC, bool STATES>
__global__ void __launch_bounds__(NT * CP, NT == 8 ? 8 : NT == 16 ? 4 : 2) k_v4_par_fwd(const Par P) {
    pdl_wait();
    pdl_trigger();
    typedef Smem<F, NT, 2, ASYNC> S;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    S &sm = *reinterpret_cast<S *>(smem_raw);
    const Place<ASYNC> L(P);
    const int c = L.c, i = L.i, T = L.T, C = L.C;
    const Copy<F, NT> cp(threadIdx.x, L.c0, C);
    const f2 w = make_float2(P.w.at(L.ch) * V4_LOG2E, P.w.at(L.ch1) * V4_LOG2E), u = mul2(L.elements((const F *)P.u), both(V4_LOG2E));
    const F *const src[2] = {(const F *)P.k + L.row, (const F *)P.v + L.row};
    if (i == 0) sm.carry[0][c] = L.ext_state(P.state_in);
    if (ASYNC) { fetch_slab<F, NT, 2>(sm, cp, 0, src, T, C, 0); cp_commit(); }
    const int n8 = (T + TK - 1) / TK, n64 = (T + COARSE - 1) / COARSE;
    const f2 W = ex2_2(w), U = ex2_2(u);
    const float range = RANGE - fmaxf(fabsf(u.x), fabsf(u.y));
    bool bad = false;       // a tile of this thread was not tame
    // FULL: every tile of the slab has its 8 tokens.  Returns false when the CTA has to start over.
    auto slab = [&](auto full_tag, int s) {
        constexpr bool FULL = decltype(full_tag)::value;
        const int t0 = s * NT * TK, mine0 = t0 + i * TK;      // first token of the slab, of this tile
        auto len = [&](int j) { return min(TK, max(0, T - t0 - j * TK)); };
        const int n = FULL ? TK : len(i);
        auto ld = [&](int tens, int j) {
            if (ASYNC) return Pair<F>::ld(&sm.slab[s & 1][tens][i * S::TILE + j * CT + 2 * c]);
            return L.ld(src[tens], (size_t)min(mine0 + j, T - 1) * C);
        };
        // the tile's own exponent (what the token-by-token maximum ends at) is its reference
        f2 e[TK];       // k, then 2^{k - reference}
        St a = empty_state();
        e[0] = mul2(ld(0, 0), both(V4_LOG2E));
        f2 kmin = e[0], kmax = e[0];
#pragma unroll
        for (int j = 0; j < TK; j++)
            if (FULL || j < n) {
                if (j > 0) e[j] = mul2(ld(0, j), both(V4_LOG2E));
                a.o = max2(add2(a.o, w), e[j]);
                kmin = min2(kmin, e[j]);
                kmax = max2(kmax, e[j]);
            }
        const f2 up = sub2(kmax, a.o), down = sub2(a.o, kmin);
        if (n > 0 && !(fmaxf(up.x, up.y) <= range && fmaxf(down.x, down.y) <= range)) bad = true;
        const f2 ref = neg2(a.o);
#pragma unroll
        for (int j = 0; j < TK; j++)
            if (FULL || j < n) {
                e[j] = ex2_2(add2(e[j], ref));
                a.p = fma2(W, a.p, mul2(e[j], ld(1, j)));
                a.q = fma2(W, a.q, e[j]);
            }
        bool stop = false;
        St x = fold_tiles<NT, false, FULL>(sm, a, sm.carry[s & 1][c], i, c, w, len, &sm.carry[(s + 1) & 1][c], bad, stop);
        if (stop) return false;
        if (n > 0) {
            if (!STATES && P.fine) L.keep(P.fine + ((size_t)L.b * n8 + mine0 / TK) * 3 * C, x);
            if (STATES && (i & 7) == 0) L.keep(P.coarse + ((size_t)L.b * n64 + mine0 / COARSE) * 3 * C, x);
        }
        if (!STATES) {
            F *y = (F *)P.y + L.row + (size_t)mine0 * C + L.ch;
            const f2 above = sub2(x.o, a.o);
            if (n > 0 && !(fmaxf(above.x, above.y) <= RANGE)) bad = true;
            const f2 sc = ex2_2(above);
            f2 p = mul2(x.p, sc), q = mul2(x.q, sc);
#pragma unroll
            for (int j = 0; j < TK; j++)
                if (FULL || j < n) {
                    const f2 v = ld(1, j), eu = mul2(U, e[j]);
                    L.st(y, mul2(fma2(eu, v, p), rcp2(add2(q, eu))));
                    y += C;
                    p = fma2(W, p, mul2(e[j], v));
                    q = fma2(W, q, e[j]);
                }
        }
        return true;
    };
    for (int s = 0; s < P.nslab; s++) {
        if (ASYNC) cp_wait0();
        __syncthreads();
        if (ASYNC && s + 1 < P.nslab) { fetch_slab<F, NT, 2>(sm, cp, (s + 1) & 1, src, T, C, (s + 1) * NT * TK); cp_commit(); }
        if (!((s + 1) * NT * TK <= T ? slab(std::true_type{}, s) : slab(std::false_type{}, s))) break;
    }
    if (__syncthreads_or(bad)) {
        if (ASYNC) cp_wait0();
        slow_forward<F, NT, ASYNC, STATES>(P, sm);
        __syncthreads();
    }
    if (!STATES && P.state_out) {
        if (i == 0) L.put_state(P.state_out, sm.carry[P.nslab & 1][c]);
    }
}

// ---------------------------------------------------------------------------------------------- backward
// The states at the start of a slab's tiles, when only coarser ones were kept: fold the summaries of the tiles between the
// kept state and the tile.  Without `coarse` there is one slab and the kept state is the initial one.
template <typename F, bool ASYNC, class S, class Len>
__device__ __noinline__ St rebuild_state(const Par &P, S &sm, const Place<ASYNC> &L, int mine0, St x, f2 w, Len len) {
    const int i = L.i, c = L.c;
    const size_t o0 = L.row + (size_t)min(mine0, L.T - 1) * L.C + L.ch, o1 = o0 - L.ch + L.ch1;
    const F *const k = (const F *)P.k, *const v = (const F *)P.v;
    const int n = len(i);
    const Slow f = slow_summary<F>(k + o0, v + o0, L.C, n, w.x), g = slow_summary<F>(k + o1, v + o1, L.C, n, w.y);
    __syncthreads();
    sm.sum[i][c] = St{make_float2(f.p, g.p), make_float2(f.q, g.q), make_float2(f.o, g.o)};
    __syncthreads();
    for (int j = P.coarse ? (i & ~7) : 0; j < i; j++) x = fold(x, mul2(w, both((float)len(j))), sm.sum[j][c]);
    __syncthreads();
    return x;
}

// As slow_forward.  gw, gu: this thread's sums.
template <typename F, int NT, bool ASYNC, bool FINE, class S>
__device__ __noinline__ void slow_walk_back(const Par &P, S &sm, f2 &gw, f2 &gu) {
    const Place<ASYNC> L(P);
    const int c = L.c, i = L.i, T = L.T, C = L.C, n8 = (T + TK - 1) / TK, n64 = (T + COARSE - 1) / COARSE, last = P.nslab - 1;
    const f2 w = make_float2(P.w.at(L.ch) * V4_LOG2E, P.w.at(L.ch1) * V4_LOG2E), u = mul2(L.elements((const F *)P.u), both(V4_LOG2E));
    const F *const k = (const F *)P.k + L.row, *const v = (const F *)P.v + L.row, *const gy = (const F *)P.gy + L.row;
    F *const gk = (F *)P.gk + L.row, *const gv = (F *)P.gv + L.row;
    if (i == 0) sm.carry[last & 1][c] = L.ext_gradient(P.gstate_out);
    gw = gu = both(0.f);
    for (int s = last; s >= 0; s--) {
        __syncthreads();
        const int t0 = s * NT * TK, mine0 = t0 + i * TK;
        auto len = [&](int j) { return min(TK, max(0, T - t0 - j * TK)); };
        const int n = len(i);
        St x;
        if (FINE) x = L.kept(P.fine + ((size_t)L.b * n8 + min(mine0 / TK, n8 - 1)) * 3 * C);
        else
            x = rebuild_state<F, ASYNC>(P, sm, L, mine0,
                                        P.coarse ? L.kept(P.coarse + ((size_t)L.b * n64 + min(mine0 / COARSE, n64 - 1)) * 3 * C) : L.ext_state(P.state_in), w, len);
        const size_t o0 = (size_t)min(mine0, T - 1) * C + L.ch, o1 = o0 - L.ch + L.ch1;
        const Slow x0{x.p.x, x.q.x, x.o.x}, x1{x.p.y, x.q.y, x.o.y}, none{0.f, 0.f, V4_MIN_VALUE};
        const SlowGrads f = slow_backward<F>(k + o0, v + o0, gy + o0, C, n, w.x, u.x, x0, none, nullptr, nullptr, 0),
                        g = slow_backward<F>(k + o1, v + o1, gy + o1, C, n, w.y, u.y, x1, none, nullptr, nullptr, 0);
        bool stop = false;
        const St e = fold_tiles<NT, true, false>(sm, St{make_float2(f.a.p, g.a.p), make_float2(f.a.q, g.a.q), make_float2(f.a.o, g.a.o)},
                                                 sm.carry[s & 1][c], i, c, w, len, &sm.carry[(s + 1) & 1][c], false, stop);
        if (n == 0) continue;
        gu = add2(gu, make_float2(f.gu, g.gu));
        gw = add2(gw, make_float2(f.gw + (e.p.x * f.dpdw + e.q.x * f.dqdw) * ex2(f.o_end + e.o.x),
                                  g.gw + (e.p.y * g.dpdw + e.q.y * g.dqdw) * ex2(g.o_end + e.o.y)));
        if (L.live) slow_backward<F>(k + o0, v + o0, gy + o0, C, n, w.x, u.x, x0, Slow{e.p.x, e.q.x, e.o.x}, gk + o0, gv + o0, C);
        if (L.live1) slow_backward<F>(k + o1, v + o1, gy + o1, C, n, w.y, u.y, x1, Slow{e.p.y, e.q.y, e.o.y}, gk + o1, gv + o1, C);
    }
}

// FINE: forward left the state at the start of every tile; else the slab's states are rebuilt from the coarse ones
// (or, one slab only, from state_in) by one more summary and fold.
template <typename F, int NT, bool ASYNC, bool FINE>
__global__ void __launch_bounds__(NT * CP, NT == 8 ? 7 : NT == 16 ? 3 : 1) k_v4_par_bwd(const Par P) {
    pdl_wait();
    pdl_trigger();
    typedef Smem<F, NT, 3, ASYNC> S;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    S &sm = *reinterpret_cast<S *>(smem_raw);
    const Place<ASYNC> L(P);
    const int c = L.c, i = L.i, T = L.T, C = L.C;
    const Copy<F, NT> cp(threadIdx.x, L.c0, C);
    const f2 w = make_float2(P.w.at(L.ch) * V4_LOG2E, P.w.at(L.ch1) * V4_LOG2E), u = mul2(L.elements((const F *)P.u), both(V4_LOG2E));
    const F *const src[3] = {(const F *)P.k + L.row, (const F *)P.v + L.row, (const F *)P.gy + L.row};
    const int n8 = (T + TK - 1) / TK, n64 = (T + COARSE - 1) / COARSE, last = P.nslab - 1;
    if (i == 0) sm.carry[last & 1][c] = L.ext_gradient(P.gstate_out);
    const float *const fine = FINE ? P.fine + (size_t)L.b * n8 * 3 * C : nullptr;
    // slab s on its way to shared memory
    auto fetch = [&](int s) {
        fetch_slab<F, NT, 3>(sm, cp, s & 1, src, T, C, s * NT * TK);
        if (FINE) fetch_states<F, NT>(sm, s & 1, fine, s * NT, n8, C, L.c0, threadIdx.x);
        cp_commit();
    };
    // the state at the start of this thread's tile (FINE) or of the 64 tokens around it, for slab s
    auto start_state = [&](int s) {
        const int t = s * NT * TK + i * TK;
        if (FINE && ASYNC) {
            auto at = [&](int r) { return *reinterpret_cast<const f2 *>(reinterpret_cast<const float *>(&sm.slab[s & 1][r][i * S::TILE + TK * CT]) + 2 * c); };
            return St{at(0), at(1), at(2)};
        }
        if (FINE) return L.kept(fine + (size_t)min(t / TK, n8 - 1) * 3 * C);
        if (P.coarse) return L.kept(P.coarse + ((size_t)L.b * n64 + min(t / COARSE, n64 - 1)) * 3 * C);
        return L.ext_state(P.state_in);
    };
    if (ASYNC) fetch(last);
    f2 gw = both(0.f), gu = both(0.f);
    const f2 W = ex2_2(w), U = ex2_2(u);
    const float range = RANGE - fmaxf(fabsf(u.x), fabsf(u.y));
    bool bad = false;
    // FULL, the result and `bad` as in forward
    auto slab = [&](auto full_tag, int s) {
        constexpr bool FULL = decltype(full_tag)::value;
        const int t0 = s * NT * TK, mine0 = t0 + i * TK;
        auto len = [&](int j) { return min(TK, max(0, T - t0 - j * TK)); };
        const int n = FULL ? TK : len(i);
        auto ld = [&](int tens, int j) {
            if (ASYNC) return Pair<F>::ld(&sm.slab[s & 1][tens][i * S::TILE + j * CT + 2 * c]);
            return L.ld(src[tens], (size_t)min(mine0 + j, T - 1) * C);
        };
        St x = start_state(s);
        if (!FINE) x = rebuild_state<F, ASYNC>(P, sm, L, mine0, x, w, len);
        // y and gy / denominator stay in registers until the gradient at the tile's end is known; k and e = 2^{k-M},
        // M = max k, are read and formed again (registers are what limits this kernel)
        f2 ys[TK], zs[TK];
        auto key = [&](int j) { return mul2(ld(0, j), both(V4_LOG2E)); };
        f2 kmin = key(0), M = kmin;
#pragma unroll
        for (int j = 1; j < TK; j++)
            if (FULL || j < n) {
                const f2 k = key(j);
                kmin = min2(kmin, k);
                M = max2(M, k);
            }
        const f2 wide = sub2(M, kmin), above = sub2(x.o, M);
        if (n > 0 && !(fmaxf(wide.x, wide.y) <= range && fmaxf(above.x, above.y) <= RANGE)) bad = true;
        f2 dpdw = both(0.f), dqdw = both(0.f);      // d(p,q)/dw since the tile's start, scaled by 2^{-M}
        St a = empty_state();
        {
            // the exponent of the gradient that leaves the tile at its start: the maximum over the tokens of j w minus
            // the exponent of the token's denominator, as the token-by-token recurrence keeps it.  Only gstate_in
            // shows which representation was used.
            if (P.gstate_in) {
                f2 o = x.o, back = both(0.f);
#pragma unroll
                for (int j = 0; j < TK; j++)
                    if (FULL || j < n) {
                        const f2 k = key(j);
                        a.o = max2(a.o, sub2(back, max2(o, add2(u, k))));
                        back = add2(back, w);
                        o = max2(add2(o, w), k);
                    }
            }
            const f2 sc = ex2_2(above), ref = neg2(M);
            f2 p = mul2(x.p, sc), q = mul2(x.q, sc);
#pragma unroll
            for (int j = 0; j < TK; j++)
                if (FULL || j < n) {
                    const f2 v = ld(1, j), e = ex2_2(add2(key(j), ref)), eu = mul2(U, e), iden = rcp2(add2(q, eu));
                    ys[j] = mul2(fma2(eu, v, p), iden);
                    zs[j] = mul2(ld(2, j), iden);
                    gw = fma2(zs[j], fma2(neg2(dqdw), ys[j], dpdw), gw);
                    gu = fma2(mul2(zs[j], eu), sub2(v, ys[j]), gu);
                    const f2 wp = mul2(W, p), wq = mul2(W, q);
                    dpdw = fma2(W, dpdw, wp); dqdw = fma2(W, dqdw, wq);
                    p = fma2(e, v, wp); q = add2(wq, e);
                    if (j & 1) no_hoist();
                }
            // the reverse recurrence from an empty gradient: exponent -M throughout
#pragma unroll
            for (int j = TK - 1; j >= 0; j--)
                if (FULL || j < n) {
                    a.p = fma2(W, a.p, zs[j]);
                    a.q = fma2(W, a.q, neg2(mul2(zs[j], ys[j])));
                }
            if (P.gstate_in) {
                const f2 r = ex2_2(sub2(ref, a.o));
                a.p = mul2(a.p, r); a.q = mul2(a.q, r);
            } else {
                a.o = ref;
            }
        }
        if (!FULL && n == 0) a = empty_state();
        bool stop = false;
        const St g = fold_tiles<NT, true, FULL>(sm, a, sm.carry[s & 1][c], i, c, w, len, &sm.carry[(s + 1) & 1][c], bad, stop);
        if (stop) return false;
        // what the gradient at the tile's end sees of the decay inside the tile
        if (FULL || n > 0) gw = fma2(fma2(g.p, dpdw, mul2(g.q, dqdw)), ex2_2(add2(M, g.o)), gw);
        const size_t out0 = L.row + (size_t)(mine0 + TK - 1) * C + L.ch;
        F *gk = (F *)P.gk + out0, *gv = (F *)P.gv + out0;
        const f2 gs = add2(g.o, M);
        if (n > 0 && !(fmaxf(gs.x, gs.y) <= GRAD_RANGE)) bad = true;
        {
            const f2 sc = ex2_2(gs), ref = neg2(M);
            f2 gp = mul2(g.p, sc), gq = mul2(g.q, sc);
#pragma unroll
            for (int j = TK - 1; j >= 0; j--) {
                if (FULL || j < n) {
                    const f2 v = ld(1, j), e = ex2_2(add2(key(j), ref)), t = mul2(zs[j], mul2(U, e));
                    L.st(gk, fma2(t, sub2(v, ys[j]), mul2(e, fma2(gp, v, gq))));
                    L.st(gv, fma2(e, gp, t));
                    gp = fma2(W, gp, zs[j]);
                    gq = fma2(W, gq, neg2(mul2(zs[j], ys[j])));
                    if (!(j & 1)) no_hoist();
                }
                gk -= C; gv -= C;
            }
        }
        return true;
    };
    for (int s = last; s >= 0; s--) {
        if (ASYNC) cp_wait0();
        __syncthreads();
        if (ASYNC && s > 0) fetch(s - 1);
        if (!((s + 1) * NT * TK <= T ? slab(std::true_type{}, s) : slab(std::false_type{}, s))) break;
    }
    if (__syncthreads_or(bad)) {
        if (ASYNC) cp_wait0();
        f2 a, e;
        slow_walk_back<F, NT, ASYNC, FINE>(P, sm, a, e);
        gw = a; gu = e;
    }
    // the tiles' shares of gw and gu, summed in a fixed order
    __syncthreads();
    sm.sum[i][c].p = gw;
    sm.sum[i][c].q = gu;
    __syncthreads();
    if (i == 0) {
        f2 a = both(0.f), e = both(0.f);
#pragma unroll 8
        for (int j = 0; j < NT; j++) { a = add2(a, sm.sum[j][c].p); e = add2(e, sm.sum[j][c].q); }
        const size_t o = (size_t)L.b * C + L.ch;
        L.st(P.gw + o, mul2(a, mul2(w, both(V4_LN2))));
        L.st(P.gu + o, e);
        if (P.gstate_in) L.put_state(P.gstate_in, sm.carry[1][c]);      // (slab 0 leaves its carry there)
    }
}

// Tiles per slab.  Longer slabs make the walk over the row shorter and the barriers fewer, and put fewer CTAs on an SM (8, 4
// or 2 of 8, 16 or 32 tiles forward; 7, 3 or 1 backward); a slab much longer than the segment is idle.  The longest that
// has its CTAs resident at once, then -- except that backward beyond 256 tokens is better off in several waves of 16 than of
// 8, which have twice the barriers and carried states per token.  us for 8 / 16 / 32 tiles, fp32, C = 2048:
//              T = 64        128           256           1024               T = 64      128          256          1024
//   fwd B = 1  3.5/4.1/4.5   5.1/4.1/4.7   8.2/5.7/4.6   26/16/11    bwd    7.2/9.5/11  7.8/4.9/5.9  14/7.3/5.9   48/22/15
//       B = 2                5.9/5.1/6.7   8.9/7.1/6.9   27/19/16                       8.6/6.5/12   15/9.1/12    60/27/31
//       B = 4  5.0/6.5/11    6.7/6.7/11    10/9.6/12     32/27/32           9.3/22/42   10/11/22     17/17/21     77/53/60
//       B = 8  6.3/11/19     8.8/11/20     14/17/21      84/87/98 *         12/32/72    14/17/38     27/28/42     199/153/189 *
// (* T = 2048.  bf16 has the same order, within a percent, at each of them.)
int pick_tiles(int B, int T, int C, bool backward) {
    const long long ctas = (long long)B * ((C + CT - 1) / CT), sms = device_sm_count();
    if (T <= 64) return 8;
    if (backward) {
        if (ctas <= sms && T > 128) return 32;
        return ctas <= 3 * sms || T > 256 ? 16 : 8;
    }
    if (ctas <= 2 * sms && T > 128) return 32;
    return ctas <= 4 * sms ? 16 : 8;
}

template <class K>
int launch(K kern, size_t smem, unsigned char (&attr_done)[64], const Par &P, int nt, cudaStream_t s) {
    if (!set_max_smem_once(kern, (int)smem, attr_done)) return WKV_ERR_LAUNCH;
    // CTAs scheduled while the kernel before drains are placed where it leaves room first: with more than one per SM that
    // is unevenly, and these kernels live from being all resident at once, so then they start together (forward and
    // backward calls of 8 x 2048 tokens x 2048 channels in turn: 193 us per call early, 143 us like this).
    const int ctas = P.B * ((P.C + CT - 1) / CT);
    return launch_kernel(ctas <= device_sm_count(), kern, dim3(ctas), dim3(nt * CP), smem, s, P);
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

// 16-byte copies and accesses of channel pairs need rows that start on 16 bytes, in every tensor; what does not is read
// and written element by element
template <typename F>
bool rows_aligned(const Par &P) {
    return (size_t)P.C * sizeof(F) % 16 == 0 && all_aligned({P.k, P.v, P.gy, P.y, P.gk, P.gv, P.gw, P.gu, P.fine, P.coarse});
}

template <typename F>
int forward_as(const Par &P, bool states, cudaStream_t s) {
    if (!rows_aligned<F>(P)) return launch_fwd<F, 16, false>(P, states, s);
    switch (pick_tiles(P.B, P.T, P.C, false)) {
        case 8: return launch_fwd<F, 8, true>(P, states, s);
        case 16: return launch_fwd<F, 16, true>(P, states, s);
        default: return launch_fwd<F, 32, true>(P, states, s);
    }
}
template <typename F>
int backward_as(Par P, float *scratch, cudaStream_t s) {
    const bool aligned = rows_aligned<F>(P) && aligned16(scratch);
    const int nt = aligned ? pick_tiles(P.B, P.T, P.C, true) : 16;
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
