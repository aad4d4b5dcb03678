// Shared pieces of the chunked tensor-core WKV kernels: tile helpers and the per-chunk
// decay bookkeeping (cumulative log-decay and the reference points that keep every
// operand scale factor inside the bf16/fp32 exponent range).
#pragma once
#include "sm100_primitives.cuh"
#include "tma_host.cuh"
#include "wkv_common.cuh"

namespace wkv {
namespace chunked {

using namespace sm100;

constexpr int CH = 64;            // tokens per chunk
constexpr int HB = 32;            // tokens per block
constexpr float LW_FLOOR = -5.298317367f;  // log(0.005)


struct __align__(16) Tile { unsigned char b[TILE_BYTES]; };

__device__ __forceinline__ uint4 ld_tile(const Tile &t, int row, int chunk) {
    return *reinterpret_cast<const uint4 *>(t.b + tile_off(row, chunk));
}
__device__ __forceinline__ void st_tile(Tile &t, int row, int chunk, const uint4 &v) {
    *reinterpret_cast<uint4 *>(t.b + tile_off(row, chunk)) = v;
}

// named barrier `id` of `threads` threads (by default the 256 compute threads of a kernel) that also ORs a predicate over them
__device__ __forceinline__ bool compute_sync_or(bool pred, int id = 1, int threads = 256) {
    uint32_t any;
    asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 q, %1, 0;\nbar.red.or.pred p, %2, %3, q;\nselp.u32 %0, 1, 0, p;\n}"
                 : "=r"(any) : "r"((uint32_t)pred), "r"(id), "r"(threads) : "memory");
    return any != 0;
}
__device__ __forceinline__ void compute_sync(int id = 1, int threads = 256) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// ---------------------------------------------------------------------------
// Per-chunk decay bookkeeping.
//
// All decay arithmetic is done in the log2 domain (one ex2 per exponential, no
// extra multiply): l2 = log2(decay) per token, c = running sum of l2 from the start
// of the thread's block, cp = c - l2.  Scale factors of neighbouring tokens differ by
// exactly one token's decay, so a thread evaluates one exponential per factor
// for its first (or last) token and walks to the others by multiplying with the
// per-token decay w = 2^{l2}.  Everything a block needs from the other block is that
// block's total, exchanged through shared memory.
constexpr float LOG2E = 1.4426950408889634f;
constexpr float LOG2_LOG2E = 0.5287663729448977f;
constexpr float LN2 = 0.6931471805599453f;
constexpr float L2_FLOOR = LW_FLOOR * LOG2E;

// log2 of the (floored) decay from the two encodings of the decay tensor; `live` tells
// whether the decay is above the floor (the floor passes no gradient)
__device__ __forceinline__ float log2_decay(float x, int w_kind, bool &live) {
    const float l2 = w_kind == WKV_W_RAW ? -exp2f(x * LOG2E) * LOG2E : x * LOG2E;
    live = l2 >= L2_FLOOR;
    return fmaxf(l2, L2_FLOOR);
}

struct Decay {           // of a thread's 4 tokens x 4 channels
    float w[4][4];   // decay of each of the tokens (1 past the segment end)
    float cp0[4];    // log2-decay accumulated from the block start to before the thread's first token
    float c3[4];     // ... up to and including its last token
    float m[4];      // ... up to and including token 15 of the block (the block midpoint reference)
    float e[4];      // the whole block
};

// Operand-pass layout for kernels with eight compute warps (256 threads):
//   warp w owns tokens 8w .. 8w+7 of the chunk (so warps 0..3 are block 0, warps 4..7 block 1);
//   lane = 16*r + 2*cc + hf:  tokens 8w + 4r .. +3,  channels 8*cc + 4*hf .. +3,
// i.e. a thread owns 4 tokens x 4 channels and reads or writes 8 bytes of a tile row at a time.
// The 16 lanes of a half-warp then cover one whole 128-byte row: free of bank conflicts.
//
// In: l2[i][ch] per-token log2-decay.  Out: l2 holds the block-local inclusive sums c; D;
// other_l2 = log2-decay total of the other block.  The totals of the eight warps go
// through `wtot` ([8][CH] floats of shared memory); `sync()` is the barrier of the 256 threads.
template <class Sync>
__device__ __forceinline__ void decay_scan8(float (&l2)[4][4], int warp, int lane, float *wtot, Decay &D,
                                            float (&other_l2)[4], Sync sync) {
    const int r = lane >> 4, ch0 = (lane & 15) * 4, blk = warp >> 2, wb = warp & 3;
    float tot[4], first[4], o[4];
#pragma unroll
    for (int ch = 0; ch < 4; ch++) {
#pragma unroll
        for (int i = 0; i < 4; i++) D.w[i][ch] = exp2f(l2[i][ch]);
        first[ch] = l2[0][ch];
    }
#pragma unroll
    for (int i = 1; i < 4; i++) vadd<4>(l2[i], l2[i], l2[i - 1]);
#pragma unroll
    for (int ch = 0; ch < 4; ch++) o[ch] = __shfl_xor_sync(0xffffffffu, l2[3][ch], 16);
    vadd<4>(tot, l2[3], o);
    if (r) *reinterpret_cast<float4 *>(wtot + warp * CH + ch0) = make_float4(tot[0], tot[1], tot[2], tot[3]);
    sync();
    const float *own = wtot + 4 * blk * CH + ch0, *oth = wtot + 4 * (blk ^ 1) * CH + ch0;
    // what lies in the block before the thread's tokens: its warp's other half and the earlier warps
    float base[4], m[4], e[4];
#pragma unroll
    for (int ch = 0; ch < 4; ch++) base[ch] = r ? o[ch] : 0.f;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const float4 a4 = *reinterpret_cast<const float4 *>(own + q * CH);
        const float4 b4 = *reinterpret_cast<const float4 *>(oth + q * CH);
        const float a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
        if (q == 0) {
#pragma unroll
            for (int ch = 0; ch < 4; ch++) { m[ch] = a[ch]; other_l2[ch] = b[ch]; }
        } else {
            vadd<4>(other_l2, other_l2, b);
            if (q == 1) {                                    // m: through token 15 of the block
                vadd<4>(m, m, a);
#pragma unroll
                for (int ch = 0; ch < 4; ch++) e[ch] = m[ch];
            } else {                                         // e: the whole block
                vadd<4>(e, e, a);
            }
        }
        if (wb > q) vadd<4>(base, base, a);
    }
#pragma unroll
    for (int i = 0; i < 4; i++) vadd<4>(l2[i], l2[i], base);
    vsub<4>(D.cp0, l2[0], first);
#pragma unroll
    for (int ch = 0; ch < 4; ch++) {
        D.c3[ch] = l2[3][ch];
        D.m[ch] = m[ch];
        D.e[ch] = e[ch];
    }
}

// Whether the chunk is "mild": no channel decays by more than 2^-128 over the whole of it, so that it can be
// factored around ONE reference point, half of the chunk's total log-decay, and the separate treatment of the pairs across
// the two blocks is not needed.  Every factor then stays within 2^+-64.  The line lies there because operands, states and gradients
// among them, are scaled by these factors, and underflow below 2^-126: values down to 2^-62 (2e-19) keep their digits, those of
// a mean loss over many tokens and products of two small ones included, and up to 2^63 nothing overflows.  (At 2^+-112 a
// state of 1e-6 was lost at 3.3 bits of decay per token.)  All threads get the same answer: every warp has
// summed the eight totals in the same order.
constexpr float MILD_L2 = -128.f;
__device__ __forceinline__ bool chunk_is_mild(const Decay &D, const float (&other_l2)[4]) {
    bool steep = false;
#pragma unroll
    for (int ch = 0; ch < 4; ch++) steep |= D.e[ch] + other_l2[ch] < MILD_L2;
    return !__any_sync(0xffffffffu, steep);
}

// What decay_scan8 gives, for a static per-channel decay (v5) and a chunk with all 64 tokens in range:
// every token of channel ch decays by lw[ch] (log2), so nothing has to be scanned or exchanged.
// w[ch] = 2^{lw[ch]}; tok0 = first of the thread's 4 tokens (0..63).
__device__ __forceinline__ void decay_static(const float (&lw)[4], const float (&w)[4], int tok0, float (&l2)[4][4],
                                             Decay &D, float (&other_l2)[4]) {
    const float t0 = (float)(tok0 & (HB - 1));
#pragma unroll
    for (int ch = 0; ch < 4; ch++) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            D.w[i][ch] = w[ch];
            l2[i][ch] = (t0 + (float)(i + 1)) * lw[ch];
        }
        D.cp0[ch] = t0 * lw[ch];
        D.c3[ch] = l2[3][ch];
        D.m[ch] = 16.f * lw[ch];
        D.e[ch] = 32.f * lw[ch];
        other_l2[ch] = D.e[ch];
    }
}

// 8-byte halves of a 16-byte tile chunk (4 bf16)
__device__ __forceinline__ void unpack4(const uint2 &q, float *f) {
    f[0] = __uint_as_float(q.x << 16); f[1] = __uint_as_float(q.x & 0xFFFF0000u);
    f[2] = __uint_as_float(q.y << 16); f[3] = __uint_as_float(q.y & 0xFFFF0000u);
}
__device__ __forceinline__ uint2 pack4(const float *f) { return make_uint2(pack2(f[0], f[1]), pack2(f[2], f[3])); }
__device__ __forceinline__ uint2 ld_tile4(const Tile &t, int row, int chunk, int half) {
    return *reinterpret_cast<const uint2 *>(t.b + tile_off(row, chunk) + 8 * half);
}
__device__ __forceinline__ void st_tile4(Tile &t, int row, int chunk, int half, const uint2 &v) {
    *reinterpret_cast<uint2 *>(t.b + tile_off(row, chunk) + 8 * half) = v;
}

// What the forward kernel hands to the backward kernels (wkv_args_t.state_ckpt):
//   sck     bf16 [B*H, nchunk+1, 64, 64]  state at the start of every chunk (key rows, value columns); of a mild
//                                         chunk times 2^m per key row
//   rhat    bf16 [B, T, C]                r_t * (decay accumulated from the chunk start to before t); of a mild chunk
//                                         times 2^-m: the operand Rt that the per-chunk backward kernel forms again, so
//                                         that the large terms of the decay gradient cancel.  (Not bit by bit: the two sum
//                                         the log-decays in another order, and about one element in 6000 is rounded to
//                                         the other side.)
//   dchunk  fp32 [B*H, nchunk, 64]        decay of each whole chunk per key channel, see ChunkDecay
//   mild    u8   [B*H * nchunk]           1 = the chunk is mild (see chunk_is_mild), 0 = steep: which body of
//                                         the per-chunk backward kernel the chunk needs
// m = c/2 rounded to a whole number, c the log2-decay of the whole chunk: the reference point that a mild chunk is
// factored around.  The states on either side of the chunk come with it, so that their products share accumulators
// (and operands) with those inside the chunk; being whole, it changes no operand's rounding on the r side.
struct CkptLayout {
    size_t sck, rhat, dchunk, mild, total;
};
inline CkptLayout ckpt_layout(int B, int T, int H) {
    const size_t n = (size_t)(T + CH - 1) / CH, bh = (size_t)B * H;
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    CkptLayout L;
    L.sck = 0;
    L.rhat = al(bh * (n + 1) * 64 * 64 * 2);
    L.dchunk = L.rhat + al((size_t)B * T * H * 64 * 2);
    L.mild = L.dchunk + al(bh * n * 64 * 4);
    L.total = L.mild + al(bh * n);
    return L;
}

// An entry of dchunk: a mild chunk's c / 2 (<= 0), a steep chunk's -c (> 0).
__device__ __forceinline__ float chunk_decay_entry(float c, bool mild) { return mild ? 0.5f * c : -c; }
__device__ __forceinline__ float pow2i(float m) { return __int_as_float((127 + __float2int_rn(m)) << 23); }   // m whole, > -127
struct ChunkDecay {
    float d;              // decay of the whole chunk
    float hs, hd, hsinv;  // scales of the states at its start and its end, 2^m and 2^{c-m}, and 2^-m (1 for a steep chunk)
};
__device__ __forceinline__ ChunkDecay chunk_decay(float entry) {
    if (entry > 0.f) return {exp2f(-entry), 1.f, 1.f, 1.f};
    const float e = exp2f(entry), m = rintf(entry);
    return {e * e, pow2i(m), exp2f(2.f * entry - m), pow2i(-m)};
}

// Time groups (see the head of wkv56_chunked.cu): G groups of L consecutive chunks per chain.
struct GroupPlan {
    int G, L;
};
constexpr int SAVE_EVERY = 8;     // chunks between two saved fp32 states (wkv_args_t.group_states)
// requested: 0 = decide from the number of chains and the device's SM count, 1 = never split,
// > 1 = that many groups (at most one per chunk)
GroupPlan plan_groups(int BH, int nchunk, int requested);
GroupPlan plan_forward(const wkv_args_t *a);

// Scratch of the time-group passes, for `units` = chains * G (all fp32; element order: see carried_at):
//   gU      [units, 64*64]   what a group adds to the state (gradient) starting from zero
//   gD      [units, 64]      decay of the whole group per key channel
//   gstart  [units, 64*64]   state (gradient) a group starts from (only where k_group_scan forms it)
struct GroupLayout {
    size_t gU, gD, gstart, total;
};
GroupLayout group_layout(size_t units);
// Up to this many groups the full pass of a group folds what the groups before it built into its starting state
// itself; with more, k_group_scan does it once for all.  The launch costs 2 to 3 us, the fold 0.13 us (forward) or
// 0.2 us (backward) per earlier group: 16 KB from L2.  (Forward / backward, folded against scanned: 40 heads, 7 groups
// 43.4 / 72.3 against 46.8 / 75.2 us; 12 heads, 24 groups 34.8 / 54.5 against 36.6 / 52.6; 1 head, 128 groups 41 / 67
// against 29 / 39.)
constexpr int GROUP_FOLD_MAX = 16;
// Element order of a matrix in gU / gstart: as the threads that carry it hold it -- thread t (0..127) has key row
// 16 (t / 32) + t % 16 and the value columns from 32 (t / 16 % 2) on, in eight quads -- so that a warp reads and
// writes consecutive 16-byte words.  (By rows, every load of a warp touched 32 lines: 0.9 us per group folded.)
__host__ __device__ __forceinline__ int carried_at(int quad, int t) { return (quad * 128 + t) * 4; }
__device__ __forceinline__ int carried_row(int e) { return 16 * (e >> 7 & 3) + (e >> 2 & 15); }
__device__ __forceinline__ int carried_col(int e) { return 32 * (e >> 6 & 1) + 4 * (e >> 9) + (e & 3); }
// quads quad0 .. quad0 + NC/4 of thread t
template <int NC>
__device__ __forceinline__ void load_carried(float (&S)[NC], const float *src, int quad0, int t) {
#pragma unroll
    for (int q = 0; q < NC / 4; q++) {
        const float4 f = *reinterpret_cast<const float4 *>(src + carried_at(quad0 + q, t));
        S[4 * q] = f.x; S[4 * q + 1] = f.y; S[4 * q + 2] = f.z; S[4 * q + 3] = f.w;
    }
}
template <int NC>
__device__ __forceinline__ void store_carried(const float (&S)[NC], float *dst, int quad0, int t) {
#pragma unroll
    for (int q = 0; q < NC / 4; q++)
        *reinterpret_cast<float4 *>(dst + carried_at(quad0 + q, t)) = make_float4(S[4 * q], S[4 * q + 1], S[4 * q + 2], S[4 * q + 3]);
}
// NC value columns from vcol0 of key row `row` of a [64,64] matrix in the caller's layout
template <int NC>
__device__ __forceinline__ void load_state_row(float (&S)[NC], const float *src, int layout, int row, int vcol0) {
    if (layout == WKV_STATE_KV) {
#pragma unroll
        for (int q = 0; q < NC / 4; q++) {
            const float4 f = *reinterpret_cast<const float4 *>(src + row * 64 + vcol0 + 4 * q);
            S[4 * q] = f.x; S[4 * q + 1] = f.y; S[4 * q + 2] = f.z; S[4 * q + 3] = f.w;
        }
    } else {
#pragma unroll
        for (int q = 0; q < NC; q++) S[q] = src[(vcol0 + q) * 64 + row];
    }
}
template <int NC>
__device__ __forceinline__ void store_state_row(const float (&S)[NC], float *dst, int layout, int row, int vcol0) {
    if (layout == WKV_STATE_KV) {
#pragma unroll
        for (int q = 0; q < NC / 4; q++)
            *reinterpret_cast<float4 *>(dst + row * 64 + vcol0 + 4 * q) = make_float4(S[4 * q], S[4 * q + 1], S[4 * q + 2], S[4 * q + 3]);
    } else {
#pragma unroll
        for (int q = 0; q < NC; q++) dst[(vcol0 + q) * 64 + row] = S[q];
    }
}
// S <- d_g S + U_g over `count` groups from unit `first` on, by `step`
template <int NC>
__device__ __forceinline__ void fold_groups(float (&S)[NC], const float *gU, const float *gD, size_t first, int step, int count,
                                            int row, int quad0, int t) {
#pragma unroll 2
    for (int i = 0; i < count; i++) {
        const size_t u = first + (ptrdiff_t)i * step;
        const float d = gD[u * 64 + row];
        float U[NC];
        load_carried<NC>(U, gU + u * 4096, quad0, t);
        vaxpy<NC>(S, d, S, U);
    }
}
int launch_group_scan(const void *group_ws, int BH, int G, const float *init, int layout, bool reverse,
                      cudaStream_t stream);

}  // namespace chunked

// How a call differs from the public one.
struct CallOpts {
    // only the wait-timeout self-test changes these: how many polls a device-side wait makes before it
    // gives up, and one TMA load that is deliberately never issued (kernel: 0 forward, 1 dS scan,
    // 2 per-chunk backward; skip_load: local chunk / step index, -1 = none)
    uint32_t wait_limit = 4000000u;
    int kernel = -1;
    int skip_load = -1;
    // status word (NULL: the first word of the workspace, cleared by the call)
    int *status = nullptr;
    // parameter gradients summed over the batch, in the parameter's element type (NULL: a->gu, a->gw)
    void *gu_sum = nullptr, *gw_sum = nullptr;
    int gu_dtype = 0, gw_dtype = 0;
};

// opt.gu_sum / gw_sum [H,64] = gu_part / gw_part [B*H, n, 64] summed over the batch and n (wkv_api.cu);
// gw_part NULL: gu alone
int fold_param_grads(const float *gu_part, const float *gw_part, int B, int H, int n, const CallOpts &opt, cudaStream_t s);

size_t chunked_group_states_bytes(const wkv_args_t *a);
// v6 with the fp32 ew = -exp(x) encoding: bytes of, and conversion into, a bf16 x tensor (a no-op otherwise)
size_t chunked_wconv_bytes(const wkv_args_t *a, bool per_token_w);
int chunked_convert_w(wkv_args_t *a, bool per_token_w, void *scratch, cudaStream_t s);
int selftest_wait(int *status, uint32_t limit, cudaStream_t s);

// `state_ckpt` (laid out as chunked::CkptLayout, or NULL) receives what the backward kernels
// reuse from the forward pass; y is not produced when `y` in `a` is NULL; `group_ws` is
// chunked::group_layout() bytes of scratch, used when the chains are split into time groups
int chunked_forward_impl(const wkv_args_t *a, bool per_token_w, void *state_ckpt, void *group_ws,
                         const CallOpts &opt, cudaStream_t s);
int chunked_forward(const wkv_args_t *a, bool per_token_w, const CallOpts &opt, cudaStream_t s);
int chunked_backward(const wkv_args_t *a, bool per_token_w, const CallOpts &opt, cudaStream_t s);

}  // namespace wkv
