// Chunked tensor-core backward of the v5/v6 WKV recurrence (bf16 I/O, fp32 state).
//
// Three kernels per BPTT segment:
//   1. the forward kernel has left (or, in a state-only mode, now writes) S_j, the state at
//      the start of every 64-token chunk (bf16), the tiles r e^{cp} and the chunk decays d_j;
//   2. k_chunk_dscan runs the reverse recurrence  D_j = d_j D_{j+1} + (r e^{cp})^T gy  with D
//      in registers and only the chunk's own product on the tensor core, writes every D_{j+1}
//      (bf16), E_j = rowsum(S_j * D_j) and the state gradient D_0;
//   3. k_chunk_bwd handles every (batch, head, chunk) independently from S_j and
//      D_{j+1}: recomputes the masked scores A, P = gy v^T, and from them the gradients, with every product on
//      tcgen05.mma.  It has two bodies.  A mild chunk (all chunks of ordinary data, see chunk_is_mild) is factored
//      around one reference point, see mild_compute.  A steep chunk takes
//         gv = A^T gy + khat D
//         gr = fr*(P~d Kt) + g*(P~x X) + e^{cp}*(gy S^T) + p_tt u k
//         gk = fk*(P~d^T Rt) + g*(P~x^T X) + e^{c_63-c}*(v D^T) + p_tt u r
//      (P~d / P~x = same-block / cross-block part of the strictly lower P; Rt, Kt, X, khat the
//      scaled operands of the forward kernel).
//
// Decay gradient.  dL/d(log w_t)[k] = w_t sum_v S_t[k,v] D_{t+1}[k,v] expands into
//   E_j + sum_{t'<=t} (a_t' + b_t') - b_t,     a = -(qrS + qrI),   b = qkD + qkI,
// where qrS/qkD are the state parts of r*gr and k*gk and qrI/qkI their intra-chunk
// parts.  The sum is a difference of large terms; it is exact only because qrI and qkI
// are built from the SAME bf16-rounded factors (Rt * (P~d Kt) and Kt * (P~d^T Rt)),
// so the common terms cancel to fp32 rounding instead of to bf16 rounding.
//
// Math reference: RWKV-v6/src/module/cuda/wkv6state_cuda_v1.cu:70-293 (what the
// gradients are), RWKV-v6/src/module/rwkv_inner.py:48-113 (the chunked form).
#include <algorithm>
#include <cfloat>
#include <cstddef>
#include <type_traits>

#include "wkv56_chunked.cuh"

namespace wkv {
namespace {

using namespace sm100;
using namespace chunked;

// ----------------------------------------------------------------------------
// dS scan

constexpr int DS_STAGES = 3;   // (four stages measured no faster: the kernel is HBM bound)

struct DscanSmem {
    Tile in[DS_STAGES][3];              // r e^{cp} and gy of the step's chunk; S at the chunk's end
    __align__(16) float dvec[DS_STAGES][CH];   // decay of the whole chunk per key channel (see ChunkDecay)
    uint64_t load_bar[DS_STAGES];       // TMA: a stage has landed
    uint64_t stage_free[DS_STAGES];     // the four scan warps are done with a stage
    uint64_t mma_bar[2];                // tensor core: a product buffer is complete
    uint64_t prod_free[2];              // the four scan warps have read a product buffer
    uint32_t tmem_base;
};

struct DscanParams {
    int T, H, nchunk, layout;
    int G, L;             // time groups per chain, chunks per group (see wkv56_chunked.cu)
    int summary;          // pass A: zero start, the only outputs are gU / gD
    const float *dchunk;  // [B*H, nchunk, 64] decay of each whole chunk (from the forward kernel, see ChunkDecay)
    const float *gstate_out;   // the caller's gradient w.r.t. the state after the segment
    const float *gstart;       // or NULL: [B*H*G, 64*64] gradient at the END of every group (order: carried_at)
    int fold;                  // pass C without gstart: start from gstate_out and the gU, gD of the groups after
    float *gstate_in;
    float *gU;                 // [B*H*G, 64*64] gradient a group builds from zero: pass A writes,
    float *gD;                 // [B*H*G, 64] decay of a whole group per key channel: pass C may read
    __nv_bfloat16 *dck;  // [B*H, nchunk+1, 64, 64]; entry j+1 = dL/dS at the end of chunk j, times the chunk's 2^{c-m}
    float *e0;           // [B*H, nchunk+1, 64]; entry j = sum_v S_j[k,v] D_j[k,v] at chunk boundary j
    int *status;
    uint32_t wait_limit;
    int skip_load;        // -1; a step index leaves that step's TMA loads out (wait-timeout test)
};

// Reverse scan of the state gradient:  D_j = d_j D_{j+1} + (r e^{cp})^T gy  over the chunks j of a
// segment, step i = 0..n-1 handling chunk j = n-1-i.  The scaled r tiles and the chunk decays
// d_j come from the forward kernel, so a step has no operand pass.
//
// Five warps.  Warp 4 (one lane) feeds the machine: TMA loads DS_STAGES steps ahead, and for every
// step the product U_j = (r e^{cp})^T gy into one of two tensor-memory buffers -- U_j does not
// depend on the carried gradient, so it is ready before the scan gets there.  Warps 0..3 carry
// D in registers (thread = key row, 32 value columns) and run the serial chain,
//   write D_{j+1} (bf16) and E_{j+1} = rowsum(S_{j+1} * D_{j+1});   D_j = d_j D_{j+1} + U_j,
// without ever synchronising with one another: each warp only waits on the barriers of the data
// it consumes and releases buffers back to warp 4.  A closing step i = n writes E_0 and D_0.
// Every wait is bounded; a warp whose wait runs out flags the status word and leaves the loop,
// which makes the waits of the others run out in turn.
//
// With time groups a CTA handles the chunks [j0, j0+n) of its chain: as a summary pass (from a
// zero gradient; no S tiles, no checkpoints, outputs gU / gD) or as the full pass from the
// gradient the group scan computed for the end of its group.  The closing step (E and D at the
// chain's first chunk boundary) belongs to the first group alone.
__global__ void __launch_bounds__(160)
k_chunk_dscan(const __grid_constant__ CUtensorMap map_rh, const __grid_constant__ CUtensorMap map_gy,
              const __grid_constant__ CUtensorMap map_s, const DscanParams P) {
    pdl_wait();
    pdl_trigger();
    extern __shared__ unsigned char smem_raw[];
    // the swizzled tiles want a 1024-byte aligned base.  The padding is added to the __shared__ array
    // itself (not to an integer copy of its address), so the compiler still knows that everything
    // behind `s` is shared memory and uses shared-memory loads and stores for the tiles.
    DscanSmem &s = *reinterpret_cast<DscanSmem *>(smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u));
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // tells the compiler it is uniform across the warp
    // one CTA per (chain, group); a summary pass leaves out group 0, which nothing needs
    const int skip = P.summary ? 1 : 0, bh = blockIdx.x / (P.G - skip), grp = blockIdx.x - bh * (P.G - skip) + skip;
    const int unit = bh * P.G + grp, b = bh / P.H, h = bh % P.H;
    const int j0 = grp * P.L, n = min(P.L, P.nchunk - j0), N = P.nchunk;
    const bool summary = P.summary != 0;
    const int nsteps = n + ((!summary && grp == 0) ? 1 : 0);    // + the closing step
    const uint32_t LIM = P.wait_limit;

    if (tid == 0) {
        for (int q = 0; q < DS_STAGES; q++) { mbar_init(&s.load_bar[q], 1); mbar_init(&s.stage_free[q], 4); }
        for (int q = 0; q < 2; q++) { mbar_init(&s.mma_bar[q], 1); mbar_init(&s.prod_free[q], 4); }
        fence_mbar_init();
    }
    if (warp == 0) { tmem_alloc(&s.tmem_base, 64); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm = __shfl_sync(0xffffffffu, s.tmem_base, 0);
    auto load_parity = [&](int i) { return (uint32_t)((i / DS_STAGES) & 1); };
    auto prod_parity = [&](int i) { return (uint32_t)((i >> 1) & 1); };
    int fail = 0;

    if (warp == 4) {
        // (the whole warp runs this, one elected lane issues)
        auto wait = [&](uint64_t *bar, uint32_t parity, uint32_t limit) { return __all_sync(0xffffffffu, mbar_wait(bar, parity, limit)) != 0; };
        int issued = -1, landed = -1, mma_issued = -1;
        auto issue_load = [&](int i) {
            if (i == P.skip_load) return;
            const int st = i % DS_STAGES, j = j0 + n - 1 - i;      // global chunk of step i
            if (elect_one()) {
                mbar_expect_tx(&s.load_bar[st], (i < n ? 2 * TILE_BYTES + CH * 4 : 0) + (summary ? 0 : TILE_BYTES));
                if (i < n) {
                    tma_load_3d(&s.in[st][0], &map_rh, &s.load_bar[st], h * 64, j * CH, b);
                    tma_load_3d(&s.in[st][1], &map_gy, &s.load_bar[st], h * 64, j * CH, b);
                    bulk_load_1d(s.dvec[st], P.dchunk + ((size_t)bh * N + j) * 64, CH * 4, &s.load_bar[st]);
                }
                if (!summary) tma_load_3d(&s.in[st][2], &map_s, &s.load_bar[st], 0, 0, bh * (N + 1) + j + 1);
            }
            issued = i;
        };
        for (int i = 0; i < DS_STAGES && i < nsteps; i++) issue_load(i);
        const uint32_t id = make_idesc(64, 32, true, true);
        for (int i = 0; i < nsteps && !fail; i++) {
            if (!wait(&s.load_bar[i % DS_STAGES], load_parity(i), LIM)) { fail = 1; break; }
            landed = i;
            if (i < n) {
                // buffer i&1 held the product of step i-2
                if (i >= 2 && !wait(&s.prod_free[i & 1], prod_parity(i - 2), LIM)) { fail = 1; break; }
                tc_fence_after();
                Tile *in = s.in[i % DS_STAGES];
                if (elect_one()) {
                    // value columns 0..31 into lanes 0..15 of each quarter, 32..63 into lanes 16..31
#pragma unroll
                    for (int hf = 0; hf < 2; hf++)
#pragma unroll
                        for (int k = 0; k < 4; k++)
                            mma_ss(tm + (hf ? (16u << 16) : 0u) + 32u * (i & 1), desc_mnmajor(&in[0], 0, k),
                                   desc_mnmajor(&in[1], 0, k) + (hf ? 4 : 0), id, k > 0);
                    mma_commit(&s.mma_bar[i & 1]);
                }
                mma_issued = i;
            }
            // the stage of step i-1 goes to step i-1+DS_STAGES as soon as the scan warps are done with it
            if (i >= 1 && i + DS_STAGES - 1 < nsteps) {
                if (!wait(&s.stage_free[(i - 1) % DS_STAGES], load_parity(i - 1), LIM)) { fail = 1; break; }
                issue_load(i + DS_STAGES - 1);
            }
        }
        if (fail) {
            // let everything in flight land before the shared and tensor memory go away
            for (int q = landed + 1; q <= issued; q++)
                if (q != P.skip_load) mbar_wait(&s.load_bar[q % DS_STAGES], load_parity(q), 200000u);
            if (mma_issued >= 0) mbar_wait(&s.mma_bar[mma_issued & 1], prod_parity(mma_issued), 100000u);
            if (mma_issued >= 1) mbar_wait(&s.mma_bar[(mma_issued - 1) & 1], prod_parity(mma_issued - 1), 100000u);
            if (P.status && lane == 0) atomicOr(P.status, 2);
        }
        __syncwarp();
    } else {
        const bool active = (lane & 16) == 0;
        const int row = warp * 16 + (lane & 15);
        const uint32_t lane_base = (uint32_t)(warp * 32);
        // U[key, value 0..31] sits in lanes 0..15 of each quarter, U[key, value 32..63] in lanes 16..31
        const int vcol0 = active ? 0 : 32;
        const size_t sbase = (size_t)bh * 64 * 64;
        float v[32];     // D, this thread's key row and half of the value columns
#pragma unroll
        for (int q = 0; q < 32; q++) v[q] = 0.f;
        if (P.gstate_out) load_state_row<32>(v, P.gstate_out + sbase, P.layout, row, vcol0);
        if (P.gstart) load_carried<32>(v, P.gstart + (size_t)unit * 4096, 0, tid);
        if (P.fold) fold_groups<32>(v, P.gU, P.gD, (size_t)bh * P.G + P.G - 1, -1, P.G - 1 - grp, row, 0, tid);
        float dprod = 1.f;      // summary pass: decay of the whole group for key channel `row`
        // 2^-m of the chunk that starts where the step's chunk ends: S_{j+1} has been scaled by 2^m
        float hinv = 1.f;
        if (!summary && j0 + n < N) hinv = chunk_decay(P.dchunk[((size_t)bh * N + j0 + n) * 64 + row]).hsinv;
        for (int i = 0; i < nsteps; i++) {
            const int st = i % DS_STAGES, j = j0 + n - 1 - i;       // global chunk of step i
            Tile *in = s.in[st];
            if (!mbar_wait(&s.load_bar[st], load_parity(i), LIM)) { fail = 1; break; }
            ChunkDecay cd = {1.f, 1.f, 1.f, 1.f};
            if (i < n) cd = chunk_decay(s.dvec[st][row]);
            // with D_{j+1} in hand: its checkpoint and E_{j+1} ...
            if (!summary) {
                f2 dot[2] = {both(0.f), both(0.f)};
#pragma unroll
                for (int c8 = 0; c8 < 4; c8++) {
                    float sv[8];
                    unpack8(ld_tile(in[2], row, (vcol0 >> 3) + c8), sv);
#pragma unroll
                    for (int q = 0; q < 8; q += 2)
                        dot[c8 & 1] = fma2(make_float2(sv[q], sv[q + 1]), make_float2(v[8 * c8 + q], v[8 * c8 + q + 1]), dot[c8 & 1]);
                }
                dot[0] = add2(dot[0], dot[1]);
                float e = dot[0].x + dot[0].y;
                e += __shfl_xor_sync(0xffffffffu, e, 16);
                if (active) P.e0[((size_t)bh * (N + 1) + (j + 1)) * 64 + row] = e * hinv;
                hinv = cd.hsinv;
            }
            if (i == n) {   // closing step: D_0 is the state gradient
                if (P.gstate_in) store_state_row<32>(v, P.gstate_in + sbase, P.layout, row, vcol0);
                break;
            }
            if (!summary) {
                uint4 *dst = reinterpret_cast<uint4 *>(P.dck + (((size_t)bh * (N + 1) + j + 1) * 64 + row) * 64 + vcol0);
#pragma unroll
                for (int c8 = 0; c8 < 4; c8++) {
                    float Dh[8];
#pragma unroll
                    for (int q = 0; q < 8; q += 2) {
                        const f2 p = mul2(both(cd.hd), make_float2(v[8 * c8 + q], v[8 * c8 + q + 1]));
                        Dh[q] = p.x; Dh[q + 1] = p.y;
                    }
                    dst[c8] = pack8(Dh);
                }
            }
            // ... then D_j = d_j D_{j+1} + U_j
            if (!mbar_wait(&s.mma_bar[i & 1], prod_parity(i), LIM)) { fail = 1; break; }
            tc_fence_after();
            {
                float u[32];
                tmem_ld16(tmem_addr(tm, lane_base, 32 * (i & 1)), u);
                tmem_ld16(tmem_addr(tm, lane_base, 32 * (i & 1) + 16), u + 16);
                tmem_ld_wait();
                dprod *= cd.d;
#pragma unroll
                for (int q = 0; q < 32; q += 2) {
                    const f2 p = fma2(both(cd.d), make_float2(v[q], v[q + 1]), mul2(both(cd.hs), make_float2(u[q], u[q + 1])));
                    v[q] = p.x; v[q + 1] = p.y;
                }
            }
            // this warp is done with the product buffer and with the stage
            tc_fence_before();
            __syncwarp();
            if (lane == 0) { mbar_arrive(&s.prod_free[i & 1]); mbar_arrive(&s.stage_free[st]); }
        }
        if (fail) {
            if (lane == 0 && P.status) atomicOr(P.status, 2);
        } else if (summary) {
            store_carried<32>(v, P.gU + (size_t)unit * 4096, 0, tid);
            if (active) P.gD[(size_t)unit * 64 + row] = dprod;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tm, 64);
}

// ----------------------------------------------------------------------------
// per-chunk gradients

enum { T_R = 0, T_K, T_V, T_W, T_GY, T_S, T_D, N_IN };

// Steep body: 14 tiles + 1 KiB.
struct SteepSmem {
    Tile in[N_IN];             // raw r, k, v, w, gy; S_j, D_{j+1}.  The w slot becomes rows
                               // 0..31 of the cumulative-decay table once w has been read.
    Tile rt, kt, x, khat;      // scaled operands
    Tile atil, ptil;           // masked scores A (with diagonal), P~
    Tile ctab_hi;              // rows 32..63 of the cumulative-decay table
    float ptt[CH];
    float kb[CH];              // decay-gradient constant of the chunk start, per channel
    __align__(16) float uf[CH];   // the head's bonus u in fp32
    uint64_t load_bar;
    uint64_t bar_early;        // P and the state products (need the raw tiles only)
    uint64_t bar_score;        // A1, A2
    uint64_t bar_grad;         // phase 2 except gv
    uint64_t bar_gv;           // gv
};

// Mild body: 13 tiles and what its threads exchange.  A chunk's tiles are refilled for the next chunk as soon as their
// last reader is done; the outputs have tiles of their own or take those of the masked scores.
struct MildSmem {
    Tile in[N_IN];             // raw r, k, v, w, gy; S', D'
    Tile rt, kt;               // scaled operands, [channel][token]
    Tile at, pt;               // masked scores A (with diagonal), P~; then gv, gw
    Tile gr, gk;
    __align__(1024) unsigned char ident[2048];   // a 16 x 16 identity in the first 32 bytes of 16 tile rows
    __align__(16) float ptt[CH];
    __align__(16) float uf[2][CH];    // the head's bonus u in fp32, by iteration parity
    __align__(16) float cst[2][2][CH];   // the chunk's entry of dchunk, K_j (see the epilogue); by iteration parity
    float dpart[2][CH];               // score diagonal, by half of the channels
    float stot[4][CH];                // per channel and run of 16 tokens: log2-decay,
    float rtot[4][CH], gup[4][CH], gwp[4][CH];   // a + b, gu, static gw
    uint64_t full[2];          // TMA: r, k, w;  v, gy, S', D'
    uint64_t turned;           // tensor core: w, r, k in tensor memory, channel by channel
    uint64_t early;            // ... P and the state parts of gr and gk
    uint64_t ops;              // compute warps: the scaled operands are in place
    uint64_t score;            // tensor core: the scores
    uint64_t mask;             // compute warps: the masked scores are in place
    uint64_t grad;             // tensor core: gr, gk
    uint64_t gv;               // ... gv
    uint64_t epi;              // compute warps: gr, gk and the turned inputs have been read
    int abort_flag;            // set by any thread whose bounded wait ran out; ends every other wait
};

constexpr int BWD_SMEM = 115712;     // half of what an SM has for one CTA; a multiple of 1024
static_assert(sizeof(SteepSmem) <= BWD_SMEM && sizeof(MildSmem) <= BWD_SMEM, "a group has 113 KiB");

// n / d for 0 <= n < 2^31 by one multiplication (Granlund and Montgomery's round-up method)
struct FastDiv {
    uint32_t mul, shift;
    FastDiv() = default;
    explicit FastDiv(uint32_t d) {
        shift = 0;
        while ((1u << shift) < d) shift++;
        mul = (uint32_t)((((uint64_t)1 << 32) * (((uint64_t)1 << shift) - d)) / d + 1);
    }
    __device__ __forceinline__ int div(int n) const { return (int)((__umulhi((uint32_t)n, mul) + (uint32_t)n) >> shift); }
};

struct BwdParams {
    int T, H, nchunk, w_kind;
    int total;           // B*H*nchunk
    FastDiv by_n, by_H;  // division by nchunk, by H
    const __nv_bfloat16 *u;
    const float *wvec;
    const float *dchunk;  // [B*H, nchunk, 64] from the forward kernel: a mild chunk's entry is its reference point
    const float *e0;  // [B*H, nchunk+1, 64]: sum_v S_j[k,v] D_j[k,v] at chunk boundary j (from the dS scan)
    float *gu_part;   // [B*H, nchunk, 64]
    float *gw_part;   // v5 only: [B*H, nchunk, 64]
    int *status;
    uint32_t wait_limit;
    int skip_load;        // -1; a chunk index whose CTAs leave their TMA loads out (wait-timeout test)
    const unsigned char *mildflag;   // [B*H*nchunk] from the forward kernel: 1 = the chunk is mild
};

// tensor-memory columns; "lo" = lanes 0..15 of each 32-lane quarter, "hi" = lanes 16..31.
// Phase 1: A1 and A2 in lo, P in hi (full 64-column score rows).  The state products of phase 1
// and everything of phase 2 are [token, 32 channels] with channels 0..31 in lo and 32..63 in hi.
enum { C_GSR = 0, C_GSK = 32,                                          // phase 1, read by the epilogue
       C_A1 = 64, C_P = 64, C_A2 = 128,                                // phase 1, read by the mask pass
       C_G1R = 64, C_G2R = 96, C_G1K = 128, C_G2K = 160, C_GV = 192,   // phase 2
       BWD_TMEM_COLS = 256 };

// fp32 cumulative log-decay table c[t][k]: rows 0..31 in `a`, rows 32..63 in `b`, 256 bytes per row;
// the 16-byte column index is XORed with (t & 7) so that 8 consecutive rows of one column fall into
// 8 different bank groups
__device__ __forceinline__ float4 *ctab_ptr4(Tile &a, Tile &b, int t, int col4) {
    return reinterpret_cast<float4 *>((t < 32 ? a.b : b.b) + (t & 31) * 256 + ((col4 ^ (t & 7)) << 4));
}
// channels 8*c8 .. +7 of row t
__device__ __forceinline__ void ld_ctab8(Tile &a, Tile &b, int t, int c8, float *v) {
    const float4 p = *ctab_ptr4(a, b, t, 2 * c8), q = *ctab_ptr4(a, b, t, 2 * c8 + 1);
    v[0] = p.x; v[1] = p.y; v[2] = p.z; v[3] = p.w;
    v[4] = q.x; v[5] = q.y; v[6] = q.z; v[7] = q.w;
}
// Sum of each of 8 values over the 16 lanes of a half-warp.  The lanes exchange halves of the
// vector (8 -> 4 -> 2 -> 1 values); lanes 2i and 2i+1 both end with the total of value i.
__device__ __forceinline__ float halving_sum8(const float *v, int l16) {
    float a4[4], a2[2];
    const bool b3 = l16 & 8, b2 = l16 & 4, b1 = l16 & 2;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float send = b3 ? v[i] : v[4 + i];
        a4[i] = (b3 ? v[4 + i] : v[i]) + __shfl_xor_sync(0xffffffffu, send, 8);
    }
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const float send = b2 ? a4[i] : a4[2 + i];
        a2[i] = (b2 ? a4[2 + i] : a4[i]) + __shfl_xor_sync(0xffffffffu, send, 4);
    }
    const float send = b1 ? a2[0] : a2[1];
    float r = (b1 ? a2[1] : a2[0]) + __shfl_xor_sync(0xffffffffu, send, 2);
    r += __shfl_xor_sync(0xffffffffu, r, 1);
    return r;
}

// The same of 4 values: lanes 4i .. 4i+3 end with the total of value i.
__device__ __forceinline__ float halving_sum4(const float *v, int l16) {
    float a2[2];
    const bool b3 = l16 & 8, b2 = l16 & 4;
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const float send = b3 ? v[i] : v[2 + i];
        a2[i] = (b3 ? v[2 + i] : v[i]) + __shfl_xor_sync(0xffffffffu, send, 8);
    }
    float r = (b2 ? a2[1] : a2[0]) + __shfl_xor_sync(0xffffffffu, b2 ? a2[0] : a2[1], 4);
    r += __shfl_xor_sync(0xffffffffu, r, 2);
    r += __shfl_xor_sync(0xffffffffu, r, 1);
    return r;
}

// The body of a steep chunk; ph: parity of the barriers' current phase; false: a wait ran out.  Eight warps: warps 0..3 and 4..7 share the four 32-lane quarters of tensor memory (warp & 3).
// The two groups split every CUDA-core phase: the operand pass by channels (4 of the 8 channels
// of a tile chunk each), the
// mask pass by score columns, the epilogue by tokens.  The decay-gradient recurrence runs forward
// in both groups; group 1 (tokens 32..63) starts from zero, parks its fp32 values in tensor-memory
// columns it has already consumed and adds the per-channel offset that group 0 publishes when it
// reaches token 31.  (Walking group 1 backward from the chunk-end constant would need no offset,
// but that constant comes from a separately rounded bf16 state and the small residuals of
// strongly decaying channels do not survive the mismatch.)
template <bool PER_TOKEN>
__device__ __forceinline__ bool
bwd_steep(const CUtensorMap &map_gr, const CUtensorMap &map_gk, const CUtensorMap &map_gv, const CUtensorMap &map_gw,
          const BwdParams &P, SteepSmem &s, const uint32_t tm, const int warp, const int bar, const int chunk_id, const uint32_t ph) {
    int lane = threadIdx.x & 31;
    asm volatile("" : "+r"(lane));      // (what follows from it is computed again for every chunk: registers)
    const int tid = 32 * warp + lane;
    const int wg = warp >> 2, w4 = warp & 3;
    const int n = P.nchunk;
    const int bh = chunk_id / n, j = chunk_id % n, b = bh / P.H, h = bh % P.H;
    const bool lo = (lane & 16) == 0;
    const int row = w4 * 16 + (lane & 15);   // accumulator row owned (token in phase 1, channel in phase 2)
    const uint32_t lane_base = (uint32_t)(w4 * 32);
    const uint32_t LIM = P.wait_limit;
    const uint32_t tm_lo = tm, tm_hi = tm + (16u << 16);

    // operand-pass coordinates (see decay_scan8): 4 tokens x 4 channels per thread, a half-warp per tile row
    const int pblk = warp >> 2, pcc = (lane & 15) >> 1, phf = lane & 1, ptok0 = 8 * warp + 4 * (lane >> 4);
    const int ch0 = pcc * 8 + 4 * phf;
    float lwc[4];
    bool livec[4];
    if (!PER_TOKEN) {
#pragma unroll
        for (int ch = 0; ch < 4; ch++) lwc[ch] = log2_decay(P.wvec[h * 64 + ch0 + ch], P.w_kind, livec[ch]);
    }
    int fail = 0;
    if (!mbar_wait(&s.load_bar, ph, LIM)) fail = 1;

    // The products that need only the raw tiles go to the tensor core before the operand pass
    // (a tcgen05.mma is issued by one thread and costs it ~100 cycles of descriptor arithmetic:
    // the accumulators of a group go out from different warps at once).
    __syncwarp();
    if (elect_one()) {
        const uint32_t id64 = make_idesc(64, 64, false, false), id32 = make_idesc(64, 32, false, false);
        if (!fail) {
            if (warp == 0) {
                // P[t,s] = sum_v gy[t,v] v[s,v]
#pragma unroll
                for (int k = 0; k < 4; k++)
                    mma_ss(tm_hi + C_P, desc_kmajor(&s.in[T_GY], 0, k), desc_kmajor(&s.in[T_V], 0, k), id64, k > 0);
            } else if (warp < 3) {
                // gr state part: GSr[t, k] = sum_v gy[t,v] S[k,v]; channels 0..31 in lo, 32..63 in hi lanes
                const int hf = warp - 1;
#pragma unroll
                for (int k = 0; k < 4; k++)
                    mma_ss((hf ? tm_hi : tm_lo) + C_GSR, desc_kmajor(&s.in[T_GY], 0, k), desc_kmajor(&s.in[T_S], 32 * hf, k), id32, k > 0);
            } else if (warp < 5) {
                // gk state part: GSk[s, k] = sum_v v[s,v] D[k,v]
                const int hf = warp - 3;
#pragma unroll
                for (int k = 0; k < 4; k++)
                    mma_ss((hf ? tm_hi : tm_lo) + C_GSK, desc_kmajor(&s.in[T_V], 0, k), desc_kmajor(&s.in[T_D], 32 * hf, k), id32, k > 0);
            }
        }
        mma_commit(&s.bar_early);
    }

    // ---------------------------------------------------------------- operand pass
    {
        float c[4][4];
        Decay D;
        unsigned livebits[4];
        // the warps' decay totals are exchanged through the first bytes of the A~ tile (unused until the mask pass)
        float *wtot = reinterpret_cast<float *>(s.atil.b);
        float other_l2[4], other[4];
        if (!PER_TOKEN && (j + 1) * CH <= P.T) {
            // static decay, whole chunk in range: closed form, nothing to scan or exchange
            float wc[4];
            unsigned lb = 0;
#pragma unroll
            for (int ch = 0; ch < 4; ch++) {
                wc[ch] = exp2f(lwc[ch]);
                lb |= (livec[ch] ? 1u : 0u) << ch;
            }
#pragma unroll
            for (int i = 0; i < 4; i++) livebits[i] = lb;
            decay_static(lwc, wc, ptok0, c, D, other_l2);
            compute_sync(bar);
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int t = ptok0 + i;
                const bool valid = j * CH + t < P.T;
                livebits[i] = 0;
                if (PER_TOKEN) {
                    float x[4];
                    unpack4(ld_tile4(s.in[T_W], t, pcc, phf), x);
#pragma unroll
                    for (int ch = 0; ch < 4; ch++) {
                        bool live;
                        const float l2 = log2_decay(x[ch], P.w_kind, live);
                        livebits[i] |= (live ? 1u : 0u) << ch;
                        c[i][ch] = valid ? l2 : 0.f;
                    }
                } else {
#pragma unroll
                    for (int ch = 0; ch < 4; ch++) {
                        livebits[i] |= (livec[ch] ? 1u : 0u) << ch;
                        c[i][ch] = valid ? lwc[ch] : 0.f;
                    }
                }
            }
            // (the barrier inside: every w value has been read, so its slot may take the table)
            decay_scan8(c, warp, lane, wtot, D, other_l2, [&] { compute_sync(bar); });
        }
        float before[4];      // log2-decay of the block before the thread's own
#pragma unroll
        for (int ch = 0; ch < 4; ch++) {
            other[ch] = exp2f(other_l2[ch]);
            before[ch] = pblk ? other_l2[ch] : 0.f;
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int t = ptok0 + i;
            float cabs[4], cv[4];      // cumulative log2-decay counted from the chunk start; its lowest mantissa
                              // bit is replaced by the "decay above the floor" flag of the token
            vadd<4>(cabs, c[i], before);
#pragma unroll
            for (int ch = 0; ch < 4; ch++)
                cv[ch] = __uint_as_float((__float_as_uint(cabs[ch]) & ~1u) | ((livebits[i] >> ch) & 1u));
            *ctab_ptr4(s.in[T_W], s.ctab_hi, t, ch0 >> 2) = make_float4(cv[0], cv[1], cv[2], cv[3]);
        }
        // r-side operands, walking forward:  fa = 2^{cp - m};  block 1 also x = r 2^{cp}  (block-local cp)
        float fa[4], fb[4];
#pragma unroll
        for (int ch = 0; ch < 4; ch++) {
            fa[ch] = exp2f(D.cp0[ch] - D.m[ch]);
            fb[ch] = exp2f(D.cp0[ch]);
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int t = ptok0 + i;
            float r[4], rt[4], xx[4];
            unpack4(ld_tile4(s.in[T_R], t, pcc, phf), r);
            vmul<4>(rt, r, fa);
            vmul<4>(fa, fa, D.w[i]);
            st_tile4(s.rt, t, pcc, phf, pack4(rt));
            if (pblk) {
#pragma unroll
                for (int ch = 0; ch < 4; ch++) {
                    xx[ch] = r[ch] * fb[ch];
                    fb[ch] *= D.w[i][ch];
                }
                st_tile4(s.x, t, pcc, phf, pack4(xx));
            }
        }
        // k-side operands, walking backward:  fa = 2^{m - c};  fb = 2^{e - c}
        //   block 0: x = k fb, khat = x 2^{total of block 1}      block 1: khat = k fb
#pragma unroll
        for (int ch = 0; ch < 4; ch++) {
            fa[ch] = exp2f(D.m[ch] - D.c3[ch]);
            fb[ch] = exp2f(D.e[ch] - D.c3[ch]);
        }
#pragma unroll
        for (int i = 3; i >= 0; i--) {
            const int t = ptok0 + i;
            float k[4], kt[4], kh[4], xx[4];
            unpack4(ld_tile4(s.in[T_K], t, pcc, phf), k);
#pragma unroll
            for (int ch = 0; ch < 4; ch++) {
                kt[ch] = k[ch] * fa[ch];
                xx[ch] = k[ch] * fb[ch];
                kh[ch] = pblk ? xx[ch] : xx[ch] * other[ch];
                fa[ch] *= D.w[i][ch];
                fb[ch] *= D.w[i][ch];
            }
            st_tile4(s.kt, t, pcc, phf, pack4(kt));
            if (!pblk) st_tile4(s.x, t, pcc, phf, pack4(xx));
            st_tile4(s.khat, t, pcc, phf, pack4(kh));
        }
    }
    fence_async_smem();
    tc_fence_before();
    const int abort1 = compute_sync_or(fail, bar);

    // ------------------------------------------------- phase 1: the scores A1, A2
    __syncwarp();
    if (elect_one()) {
        if (!abort1) {
            tc_fence_after();
            if (warp == 0) {
                const uint32_t id64 = make_idesc(64, 64, false, false);
#pragma unroll
                for (int k = 0; k < 4; k++)
                    mma_ss(tm_lo + C_A1, desc_kmajor(&s.rt, 0, k), desc_kmajor(&s.kt, 0, k), id64, k > 0);
            } else if (warp == 1) {
                const uint32_t id32 = make_idesc(64, 32, false, false);
#pragma unroll
                for (int k = 0; k < 4; k++)
                    mma_ss(tm_lo + C_A2, desc_kmajor(&s.x, 0, k), desc_kmajor(&s.x, 0, k), id32, k > 0);
            }
        }
        mma_commit(&s.bar_score);
    }
    // meanwhile: the bonus term of the score diagonal, sum_k r_t u k_t, in the warps whose 16 rows x
    // 32 columns straddle the diagonal; the lo lane takes channels 0..31 of the row, the hi lane 32..63
    const int col0 = 32 * wg;                       // score columns this group masks
    const bool diag_warp = (w4 >= 2) == (wg == 1), cross_warp = wg == 0 && w4 >= 2;
    float diag = 0.f;
    if (diag_warp) {
        f2 d2 = both(0.f);
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int c8 = (lo ? 0 : 4) + c;
            float a[8], d[8], uq[8];
            unpack8(ld_tile(s.in[T_R], row, c8), a);
            unpack8(ld_tile(s.in[T_K], row, c8), d);
            {
                const float4 u0 = *reinterpret_cast<const float4 *>(s.uf + 8 * c8), u1 = *reinterpret_cast<const float4 *>(s.uf + 8 * c8 + 4);
                uq[0] = u0.x; uq[1] = u0.y; uq[2] = u0.z; uq[3] = u0.w; uq[4] = u1.x; uq[5] = u1.y; uq[6] = u1.z; uq[7] = u1.w;
            }
#pragma unroll
            for (int q = 0; q < 8; q += 2)
                d2 = fma2(mul2(make_float2(a[q], a[q + 1]), make_float2(uq[q], uq[q + 1])), make_float2(d[q], d[q + 1]), d2);
        }
        diag = d2.x + d2.y;
        diag += __shfl_xor_sync(0xffffffffu, diag, 16);
    }
    if (!abort1 && !(mbar_wait(&s.bar_early, ph, LIM) && mbar_wait(&s.bar_score, ph, LIM))) fail = 1;
    tc_fence_after();

    // mask pass: lo lanes build A~ (row t), hi lanes build P~ (row t); this group's 32 columns.
    // P~ is split: its two same-block triangles go to the P~ tile (cross block zero), the
    // cross block (t >= 32, s < 32) to the same rows of the v tile, whose readers are done.
    {
        const int t = row;
        float a[32];
        // columns col0..+31 of A1 (lo lanes) and of P (hi lanes) share their tensor-memory columns
        if (diag_warp || cross_warp) {
            tmem_ld16(tmem_addr(tm, lane_base, C_A1 + col0), a);
            tmem_ld16(tmem_addr(tm, lane_base, C_A1 + col0 + 16), a + 16);
        }
        if (cross_warp) {           // rows 32..63, columns 0..31: every entry kept; A~ takes the cross-block scores from their own product
#pragma unroll
            for (int q4 = 0; q4 < 8; q4++) {
                float a2[4];
                tmem_ld4(tmem_addr(tm, lane_base, C_A2 + 4 * q4), a2);
                tmem_ld_wait();
#pragma unroll
                for (int q = 0; q < 4; q++) a[4 * q4 + q] = lo ? a2[q] : a[4 * q4 + q];
            }
        } else if (diag_warp) {
            tmem_ld_wait();
            // local row lim = t - col0: columns below it are kept, column lim is the diagonal (the bonus
            // term in A~, p_tt set aside and zero in P~).  Rows 0..15 of the block cannot reach columns
            // 16..31, rows 16..31 keep all of columns 0..15.
            const float dval = lo ? diag : 0.f;
            float pt = 0.f;
            if ((w4 & 1) == 0) {
                const int lim = t - col0;
#pragma unroll
                for (int q = 0; q < 16; q++) {
                    if (q == lim) pt = a[q];
                    a[q] = q < lim ? a[q] : (q == lim ? dval : 0.f);
                    a[16 + q] = 0.f;
                }
            } else {
                const int lim = t - col0 - 16;
#pragma unroll
                for (int q = 0; q < 16; q++) {
                    if (q == lim) pt = a[16 + q];
                    a[16 + q] = q < lim ? a[16 + q] : (q == lim ? dval : 0.f);
                }
            }
            if (!lo) s.ptt[t] = pt;
        } else {                    // upper-right block: nothing survives
#pragma unroll
            for (int q = 0; q < 32; q++) a[q] = 0.f;
        }
        Tile &dst = lo ? s.atil : (cross_warp ? s.in[T_V] : s.ptil);
#pragma unroll
        for (int c8 = 0; c8 < 4; c8++) st_tile(dst, t, (col0 >> 3) + c8, pack8(a + 8 * c8));
        if (cross_warp && !lo) {
#pragma unroll
            for (int c8 = 0; c8 < 4; c8++) st_tile(s.ptil, t, c8, make_uint4(0u, 0u, 0u, 0u));
        }
    }
    fence_async_smem();
    tc_fence_before();
    const int abort2 = compute_sync_or(fail, bar) | abort1;

    // ------------------------------------------------- phase 2: token-major accumulators
    // every accumulator is [token, 32 channels]: channels 0..31 in the lo lanes, 32..63 in the hi lanes
    // gv is needed last: it goes to a barrier of its own, from the two warps that have no gradient
    // product to issue (so that no warp enters the epilogue later than the others).
    __syncwarp();
    if (elect_one()) {
        tc_fence_after();
        const uint32_t id_kn = make_idesc(64, 32, false, true), id_nn = make_idesc(64, 32, true, true);
        const int hf = warp & 1;
        const uint32_t tmh = hf ? tm_hi : tm_lo;
        const uint64_t boff = hf ? 4 : 0;     // +64 bytes: the upper 32 of the 64 contiguous elements
        if (abort2) {
            mma_commit(&s.bar_grad);          // nothing is issued
        } else if (warp == 0) {
            // gr intra, across blocks: G2r[t >= 32, k] = sum_{s<32} P~x[t,s] X[s,k]   (rows t < 32 are not read)
#pragma unroll
            for (int hq = 0; hq < 2; hq++)
#pragma unroll
                for (int k = 0; k < 2; k++)
                    mma_ss((hq ? tm_hi : tm_lo) + C_G2R, desc_kmajor(&s.in[T_V], 0, k),
                           desc_mnmajor(&s.x, 0, k) + (hq ? 4 : 0), id_kn, k > 0);
            mma_commit(&s.bar_grad);
        } else if (warp == 1) {
            // gk intra, across blocks: G2k[s < 32, k] = sum_{t>=32} P~x[t,s] X[t,k]   (rows s >= 32 are not read)
#pragma unroll
            for (int hq = 0; hq < 2; hq++)
#pragma unroll
                for (int k = 0; k < 2; k++)
                    mma_ss((hq ? tm_hi : tm_lo) + C_G2K, desc_mnmajor(&s.in[T_V], 32, k),
                           desc_mnmajor(&s.x, 32, k) + (hq ? 4 : 0), id_nn, k > 0);
            mma_commit(&s.bar_grad);
        } else if (warp == 2 || warp == 3) {
            // gr intra, same block: G1r[t,k] = sum_s P~d[t,s] Kt[s,k]
#pragma unroll
            for (int k = 0; k < 4; k++)
                mma_ss(tmh + C_G1R, desc_kmajor(&s.ptil, 0, k), desc_mnmajor(&s.kt, 0, k) + boff, id_kn, k > 0);
            mma_commit(&s.bar_grad);
        } else if (warp == 4 || warp == 5) {
            // gk intra, same block: G1k[s,k] = sum_t P~d[t,s] Rt[t,k]
#pragma unroll
            for (int k = 0; k < 4; k++)
                mma_ss(tmh + C_G1K, desc_mnmajor(&s.ptil, 0, k), desc_mnmajor(&s.rt, 0, k) + boff, id_nn, k > 0);
            mma_commit(&s.bar_grad);
        } else {
            mma_commit(&s.bar_grad);
        }
        if (!abort2 && warp >= 6) {
            // gv[s, v] = sum_t A~[t,s] gy[t,v] + sum_k khat[s,k] D[k,v]
#pragma unroll
            for (int k = 0; k < 4; k++)
                mma_ss(tmh + C_GV, desc_mnmajor(&s.atil, 0, k), desc_mnmajor(&s.in[T_GY], 0, k) + boff, id_nn, k > 0);
#pragma unroll
            for (int k = 0; k < 4; k++)
                mma_ss(tmh + C_GV, desc_kmajor(&s.khat, 0, k), desc_mnmajor(&s.in[T_D], 0, k) + boff, id_kn, true);
        }
        mma_commit(&s.bar_gv);
    }

    // ------------------------------------------------- epilogue
    // A thread owns token t = row and the 32 channels of its lane half; group 0 is the gr side,
    // group 1 the gk side.  While gv is still being accumulated (from A~, gy, khat, D) only tiles
    // outside that product are touched: gr and gk are staged in place of the scaled operands each
    // thread has just consumed (gr->rt, gk->kt), S and the P~ tile carry the exchange between the
    // groups, the v tile the per-warp sums.  Once gv is done: gv->gy, gw->D.
    Tile &o_gr = s.rt, &o_gk = s.kt, &o_gw = s.in[T_D], &o_gv = s.in[T_GY];
    Tile &ct_lo = s.in[T_W], &ct_hi = s.ctab_hi;
    int le = lane;
    asm volatile("" : "+r"(le));
    const int hh = le >> 4, l16 = le & 15, t = w4 * 16 + l16;
    const float ptt_t = s.ptt[t];
    const bool tvalid = j * CH + t < P.T;
    // [NPART][64] totals of the token scan, and as many partial sums for gu / the static gw: per 16 tokens, in the v tile
    constexpr int NPART = 4;
    float *wtot = reinterpret_cast<float *>(s.in[T_V].b);
    float *gup = wtot + NPART * CH, *gwp = gup + NPART * CH;

    // decay-gradient constant sum_v S[k,v] D[k,v] at the chunk start (consumed after two more barriers)
    if (tid < CH) s.kb[tid] = P.e0[((size_t)bh * (n + 1) + j) * 64 + tid];
    if (!abort2 && !mbar_wait(&s.bar_grad, ph, LIM)) fail = 1;
    tc_fence_after();

    // The decay gradient of token t is  glw_t = K_j + sum_{t'<=t} (a_t' + b_t') - b_t  with
    //   a_t = -(qrS_t + qrI_t)   (gr side),     b_t = qkD_t + qkI_t   (gk side),
    // qrS/qkD the state parts of r*gr and k*gk and qrI/qkI their intra-chunk parts (file header).
    // Compiled for each side.  (One code for both, with 8-byte accesses of the tiles: an all-steep 7B segment 865 us, this 822.)
    auto side_pass = [&](auto side) {
        constexpr bool GR = decltype(side)::value;
        constexpr float sg = GR ? 1.f : -1.f;
        const bool has2 = GR == (w4 >= 2);                    // the cross-block accumulator covers this token
        const Tile &t_own = GR ? s.rt : s.kt;
        const Tile &t_raw = GR ? s.in[T_R] : s.in[T_K], &t_oth = GR ? s.in[T_K] : s.in[T_R];
        const int cGS = GR ? C_GSR : C_GSK, cG1 = GR ? C_G1R : C_G1K, cG2 = GR ? C_G2R : C_G2K;
        Tile &o_main = GR ? o_gr : o_gk;
        Tile &exch = GR ? s.in[T_S] : s.ptil;                 // what the other group needs from this one
        const int zrow = GR ? t - 1 : t;                      // gr factors use c_{t-1}, gk factors c_t
        const int mrow = t < HB ? 15 : 47;                    // row of the table that holds the reference point
        // four channels at a time: 4 c4 .. +3; the tiles 16 bytes at a time (8-byte accesses of a column of rows find half
        // of the banks), but for one of the three: its registers would be spilled
#pragma unroll 1
        for (int bt8 = 0; bt8 < 4; bt8++) {
            const int c8 = 4 * hh + bt8;
            const uint4 own8 = ld_tile(t_own, t, c8), raw8 = ld_tile(t_raw, t, c8);
            uint4 out8;
#pragma unroll
            for (int half = 0; half < 2; half++) {
                const int bt = 2 * bt8 + half, c4 = 8 * hh + bt;
                auto of8 = [&](const uint4 &q) { return half ? make_uint2(q.z, q.w) : make_uint2(q.x, q.y); };
                float g1[4], gs[4], g2[4];
                tmem_ld4(tmem_addr(tm, lane_base, cG1 + 4 * bt), g1);
                tmem_ld4(tmem_addr(tm, lane_base, cGS + 4 * bt), gs);
                if (has2) tmem_ld4(tmem_addr(tm, lane_base, cG2 + 4 * bt), g2);
                auto get4 = [](float *v, const float4 &f) { v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w; };
                float own[4], raw[4], oth[4], uu[4], z[4], f1[4], fS[4], out[4], ab[4];
                get4(z, zrow >= 0 ? *ctab_ptr4(ct_lo, ct_hi, zrow, c4) : make_float4(0.f, 0.f, 0.f, 0.f));
                get4(f1, *ctab_ptr4(ct_lo, ct_hi, mrow, c4));
                get4(fS, *ctab_ptr4(ct_lo, ct_hi, 63, c4));
                get4(uu, *reinterpret_cast<const float4 *>(s.uf + 4 * c4));
                unpack4(of8(own8), own);
                unpack4(of8(raw8), raw);
                unpack4(ld_tile4(t_oth, t, c8, half), oth);
                tmem_ld_wait();
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    f1[q] = exp2f(sg * (z[q] - f1[q]));
                    fS[q] = exp2f(GR ? z[q] : fS[q] - z[q]);
                }
                // (the r side's state part from r e^{cp} as the dS scan had it, rounded: E_j then cancels against it.  Unrounded,
                // the sum over the tokens that is a static decay's gradient was 2 to 4 % off, with it 0.5)
                vmul<4>(ab, raw, fS);
                if (GR) unpack4(pack4(ab), ab);
                vmul<4>(ab, ab, gs);
                vmul<4>(fS, fS, gs);
                vfma<4>(out, f1, g1, fS);
                vfma<4>(ab, own, g1, ab);
                vmul<4>(uu, uu, oth);
                vaxpy<4>(out, ptt_t, uu, out);
                if (has2) {
                    float xx[4], e0r[4];
                    unpack4(ld_tile4(s.x, t, c8, half), xx);
                    get4(e0r, *ctab_ptr4(ct_lo, ct_hi, 31, c4));
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        out[q] += exp2f(sg * (z[q] - e0r[q])) * g2[q];
                        ab[q] += xx[q] * g2[q];
                    }
                }
                {
                    const uint2 o = pack4(out);
                    if (half) { out8.z = o.x; out8.w = o.y; } else { out8.x = o.x; out8.y = o.y; }
                }
#pragma unroll
                for (int q = 0; q < 4; q++) ab[q] *= -sg;
                if (GR == (bt < 4)) {       // kept, in columns that have just been read
                    tmem_st4(tmem_addr(tm, lane_base, cGS + 4 * bt), ab);
                } else {
                    *reinterpret_cast<float4 *>(exch.b + tile_off(t, 4 * hh + (bt & 3))) = make_float4(ab[0], ab[1], ab[2], ab[3]);
                }
                if (!GR) {
                    // gu: sum over this warp's 16 tokens of p_tt r k, by a halving exchange
                    float gue[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) gue[q] = ptt_t * raw[q] * oth[q];
                    const float tot = halving_sum4(gue, l16);
                    if ((l16 & 3) == 0) gup[w4 * CH + 4 * c4 + (l16 >> 2)] = tot;
                }
            }
            st_tile(o_main, t, c8, out8);
        }
        tmem_st_wait();
    };
    if (wg == 0) side_pass(std::true_type{}); else side_pass(std::false_type{});
    {
        // gv: accumulator [s, v]; each group takes half of the columns
        if (!abort2 && !mbar_wait(&s.bar_gv, ph, LIM)) fail = 1;
        tc_fence_after();
        float gv[16];
        tmem_ld16(tmem_addr(tm, lane_base, C_GV + 16 * wg), gv);
        tmem_ld_wait();
#pragma unroll
        for (int c8 = 0; c8 < 2; c8++) st_tile(o_gv, t, 4 * hh + 2 * wg + c8, pack8(gv + 8 * c8));
    }
    compute_sync(bar);
    // the token scan of z = a + b for this thread's 16 channels: 32*hh + 16*wg .. +15
    float bsub[16], keep[16];   // keep: a_t (group 0), b_t (group 1) of these channels; then z_t
    tmem_ld16(tmem_addr(tm, lane_base, wg ? C_GSK + 16 : C_GSR), keep);
    tmem_ld_wait();
    {
        const Tile &got = wg ? s.in[T_S] : s.ptil;         // what the other group left for this one
#pragma unroll
        for (int c4 = 0; c4 < 4; c4++) {
            const float4 o = *reinterpret_cast<const float4 *>(got.b + tile_off(t, 4 * hh + c4));
            const float ov[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int i = 4 * c4 + q;
                bsub[i] = wg ? keep[i] : ov[q];            // b_t
                keep[i] += ov[q];                          // z_t
            }
        }
#pragma unroll
        for (int off = 1; off < 16; off <<= 1) {
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const float o = __shfl_up_sync(0xffffffffu, keep[i], off, 16);
                if (l16 >= off) keep[i] += o;
            }
        }
        if (l16 == 15) {
#pragma unroll
            for (int c4 = 0; c4 < 4; c4++)
                *reinterpret_cast<float4 *>(wtot + w4 * CH + 32 * hh + 16 * wg + 4 * c4) =
                    make_float4(keep[4 * c4], keep[4 * c4 + 1], keep[4 * c4 + 2], keep[4 * c4 + 3]);
        }
    }
    compute_sync(bar);
    {
        const int kb0 = 32 * hh + 16 * wg;                 // first of the 16 channels
        float glw[16];
        // the constant of the chunk start plus the earlier warps' totals
#pragma unroll
        for (int c4 = 0; c4 < 4; c4++) {
            float4 o = *reinterpret_cast<const float4 *>(s.kb + kb0 + 4 * c4);
            for (int w = 0; w < w4; w++) {
                const float4 p = *reinterpret_cast<const float4 *>(wtot + w * CH + kb0 + 4 * c4);
                o.x += p.x; o.y += p.y; o.z += p.z; o.w += p.w;
            }
            glw[4 * c4] = o.x + keep[4 * c4] - bsub[4 * c4];
            glw[4 * c4 + 1] = o.y + keep[4 * c4 + 1] - bsub[4 * c4 + 1];
            glw[4 * c4 + 2] = o.z + keep[4 * c4 + 2] - bsub[4 * c4 + 2];
            glw[4 * c4 + 3] = o.w + keep[4 * c4 + 3] - bsub[4 * c4 + 3];
        }
        if (PER_TOKEN) {
            // times the floored log-decay of the token, zero where the floor was hit (no gradient)
#pragma unroll
            for (int c2 = 0; c2 < 2; c2++) {
                const int c8 = (kb0 >> 3) + c2;
                float c[8], cp[8];
                ld_ctab8(ct_lo, ct_hi, t, c8, c);
                if (t > 0) {
                    ld_ctab8(ct_lo, ct_hi, t - 1, c8, cp);
                } else {
#pragma unroll
                    for (int q = 0; q < 8; q++) cp[q] = 0.f;
                }
                float o[8];
#pragma unroll
                for (int q = 0; q < 8; q++)
                    o[q] = (__float_as_uint(c[q]) & 1u) ? glw[8 * c2 + q] * (c[q] - cp[q]) * LN2 : 0.f;
                st_tile(o_gw, t, c8, pack8(o));
            }
        } else {
#pragma unroll
            for (int c2 = 0; c2 < 2; c2++) {
                float e[8];
#pragma unroll
                for (int q = 0; q < 8; q++) e[q] = tvalid ? glw[8 * c2 + q] : 0.f;
                const float tot = halving_sum8(e, l16);
                if ((l16 & 1) == 0) gwp[w4 * CH + kb0 + 8 * c2 + (l16 >> 1)] = tot;
            }
        }
    }
    fence_async_smem();
    tc_fence_before();
    const int abort3 = compute_sync_or(fail, bar) | abort2;
    if (!abort3 && tid == 0) {
        tma_store_3d(&map_gr, &o_gr, h * 64, j * CH, b);
        tma_store_3d(&map_gk, &o_gk, h * 64, j * CH, b);
        tma_store_3d(&map_gv, &o_gv, h * 64, j * CH, b);
        if (PER_TOKEN) tma_store_3d(&map_gw, &o_gw, h * 64, j * CH, b);
        tma_store_commit();
    }
    // per-chunk partials, folded later in a fixed order
    if (tid >= 64 && tid < 128) {
        const int k = tid - 64;
        float tot = gup[k];
#pragma unroll
        for (int q = 1; q < NPART; q++) tot += gup[q * CH + k];
        P.gu_part[((size_t)bh * n + j) * 64 + k] = tot;
    } else if (!PER_TOKEN && tid >= 128 && tid < 192) {
        const int k = tid - 128;
        bool live;
        const float lw = log2_decay(P.wvec[h * 64 + k], P.w_kind, live) * LN2;
        float tot = gwp[k];
#pragma unroll
        for (int q = 1; q < NPART; q++) tot += gwp[q * CH + k];
        P.gw_part[((size_t)bh * n + j) * 64 + k] = live ? tot * lw : 0.f;
    }
    if (!abort3 && tid == 0) tma_store_wait_read();   // the tiles must outlive the reads of the bulk stores
    if (abort3 && tid == 0) {
        // every warp has arrived on every barrier: whatever was issued is done once they complete
        mbar_wait(&s.bar_early, ph); mbar_wait(&s.bar_score, ph); mbar_wait(&s.bar_grad, ph); mbar_wait(&s.bar_gv, ph);
        if (j != P.skip_load) mbar_wait(&s.load_bar, ph, 200000u);
        if (P.status) atomicOr(P.status, 4);
    }
    return abort3 == 0;
}

// ----------------------------------------------------------------------------
// The body of a mild chunk.
//
// With m (half of the chunk's log2-decay c, see CkptLayout) as the one reference point, Rt = r 2^{cp-m},
// Kt = k 2^{m-c_t}, and S' = 2^m S, D' = 2^{c-m} D as the forward kernel and the dS scan have left them:
//   Gr = P~ Kt + gy S'^T        gr = 2^{cp-m} Gr + p_tt u k       -a = Rt * Gr
//   Gk = P~^T Rt + v D'^T       gk = 2^{m-c_t} Gk + p_tt u r       b = Kt * Gk
//   gv = A~^T gy + Kt D'
// one accumulator and one factor per side.
//
// What bounds a chunk's CUDA-core work is the number of instructions, so everything elementwise is done by threads
// that own one channel and 16 consecutive tokens: the decay sums, the factors, the gradients and the token scan of the
// decay gradient are then serial code on registers, with no shuffles, no table of sums and nothing to read again
// by other threads (78 instructions per 32 elements, where threads of 4 x 4 elements and of one token took 129).
// Inputs come [token][channel]; the tensor core turns them: w, r, k times a 16 x 16 identity, exact in
// fp32, and a thread reads its 16 values with one tcgen05.ld.  (An infinite one, times the identity's zeros, spoils
// the other 15 of its run: the chunk is then read from the tiles, see mild_inputs_again.)  All accumulators are
// [channel][token] likewise, read by the 16-lane load (tmem_ld16_split32), which covers an M = 64, N = 64 accumulator with all threads: no product
// is cut into column halves.  gr, gk and gw go back to [token][channel] by 2-byte stores.
//
// Eight compute warps (w4 = warp & 3: channels 16 w4 .. +15; lane & 15: the channel; tokens 32 (lane >> 4) +
// 16 (warp >> 2) .. +15) walk over the group's chunks, and a feeder warp issues every load, a chunk ahead, and every
// tcgen05.mma.  (One chunk per CTA, two CTAs on an SM: of 15.6 k cycles per chunk 8 k went to the start of the CTA, its
// first loads and the drain of its stores.)
// 4 rows of 4096 tokens x 64 heads: 505 us with one CTA per chunk and the 4 x 4 threads, 400 with this arithmetic, 304
// with both; what is left is spread over waits for products (2.3 k of 9.1 k cycles per chunk and group), issue (50 %)
// and shared memory (46 % of its cycles).
//
// Tensor memory, 64 columns each, lo lanes / hi lanes:
enum { U_WR = 0,      // w turned (then the log2-decays summed up to each token, less m) / r turned
       U_KV = 64,     // k turned / gv [token][value]
       U_AP = 128,    // A / P, [t][s]
       U_G = 192 };   // Gr / Gk, [channel][token]

// Every stride-th chunk from `first` on, of one kind.  All lanes of a warp walk together.
struct ChunkWalk {
    const unsigned char *flag;     // [total]
    int at, stride, total;         // the 32 chunks from `at` on
    unsigned kind, left;           // left: which of them are still to come
    __device__ __forceinline__ void fetch() {
        const int c = at + (int)(threadIdx.x & 31) * stride;
        left = __ballot_sync(0xffffffffu, c < total && (flag[c] != 0) == (kind != 0));
    }
    __device__ __forceinline__ ChunkWalk(const unsigned char *f, int first, int step, int n, unsigned k)
        : flag(f), at(first), stride(step), total(n), kind(k) { fetch(); }
    __device__ __forceinline__ int next() {      // -1: no more
        while (left == 0) {
            at += 32 * stride;
            if (at >= total) return -1;
            fetch();
        }
        const int q = __ffs(left) - 1;
        left &= left - 1;
        return at + q * stride;
    }
};

// The feeder of a group's mild chunks, every stride-th from `first` on: loads and products, by one lane.  A tile is loaded for
// the next chunk as soon as the current one is done with it: w, r, k when the operands are in place, v and S' when P and
// the state products are done, gy and D' when gv is.  false: a wait ran out.
template <bool PER_TOKEN>
__device__ __forceinline__ bool
mild_feed(const CUtensorMap &map_r, const CUtensorMap &map_k, const CUtensorMap &map_v, const CUtensorMap &map_w,
         const CUtensorMap &map_gy, const CUtensorMap &map_s, const CUtensorMap &map_d,
          const BwdParams &P, MildSmem &s, const uint32_t tm, const int first, const int stride) {
    const int n = P.nchunk;
    const uint32_t LIM = P.wait_limit, tm_hi = tm + (16u << 16);
    // (the whole warp runs this, one elected lane issues)
    auto wait = [&](uint64_t *bar, uint32_t ph) {
        if (__all_sync(0xffffffffu, mbar_wait_or_abort(bar, ph, &s.abort_flag, LIM))) return true;
        *reinterpret_cast<volatile int *>(&s.abort_flag) = 1;
        return false;
    };
    ChunkWalk walk(P.mildflag, first, stride, P.total, 1u);
    int chunk = walk.next();
    if (chunk < 0) return true;
    struct At { int c, h, t0, b, s; };
    auto at = [&](int c) { const int bh = P.by_n.div(c), j = c - bh * n, b = P.by_H.div(bh); return At{c, (bh - b * P.H) * 64, j * CH, b, bh * (n + 1) + j}; };
    auto load0 = [&](const At &x, uint32_t ph) {
        mbar_expect_tx(&s.full[0], (PER_TOKEN ? 3 : 2) * TILE_BYTES + 2 * CH * 4);
        bulk_load_1d(s.cst[ph][0], P.dchunk + (size_t)x.c * CH, CH * 4, &s.full[0]);
        bulk_load_1d(s.cst[ph][1], P.e0 + (size_t)x.s * CH, CH * 4, &s.full[0]);
        if (PER_TOKEN) tma_load_3d(&s.in[T_W], &map_w, &s.full[0], x.h, x.t0, x.b);
        tma_load_3d(&s.in[T_R], &map_r, &s.full[0], x.h, x.t0, x.b);
        tma_load_3d(&s.in[T_K], &map_k, &s.full[0], x.h, x.t0, x.b);
    };
    auto load1a = [&](const At &x) {
        mbar_expect_tx(&s.full[1], 4 * TILE_BYTES);
        tma_load_3d(&s.in[T_V], &map_v, &s.full[1], x.h, x.t0, x.b);
        tma_load_3d(&s.in[T_S], &map_s, &s.full[1], 0, 0, x.s);
        tma_prefetch_l2_3d(&map_gy, x.h, x.t0, x.b);
        tma_prefetch_l2_3d(&map_d, 0, 0, x.s + 1);
    };
    auto load1b = [&](const At &x) {
        tma_load_3d(&s.in[T_GY], &map_gy, &s.full[1], x.h, x.t0, x.b);
        tma_load_3d(&s.in[T_D], &map_d, &s.full[1], 0, 0, x.s + 1);
    };
    // (a chunk whose loads are left out on the host's word: the wait-timeout test)
    auto skip = [&](int c) { return c - P.by_n.div(c) * n == P.skip_load; };
    bool loads = !skip(chunk);         // the current chunk's have been issued
    if (loads) {
        const At x = at(chunk);
        if (elect_one()) { load0(x, 0); load1a(x); load1b(x); }
    }
    bool fine = true;
    for (uint32_t ph = 0; chunk >= 0 && fine; ph ^= 1) {
        const int next = walk.next();
        const bool more = next >= 0 && !skip(next);
        const At x = at(next >= 0 ? next : chunk);
        int stage = 0;       // barriers committed to
        bool all = !more;    // the next chunk's loads have all been issued
        // operand descriptors: that of the structure's first tile plus an offset
        const uint64_t d0 = make_desc(smem_u32(&s));
        auto kmaj = [&](uint32_t off, int k16) { return d0 + ((off + 32 * k16) >> 4); };
        auto mnmaj = [&](uint32_t off, int k16) { return d0 + ((off + 16 * TILE_ROW_BYTES * k16) >> 4); };
        do {
            if (!wait(&s.full[0], ph)) break;
            tc_fence_after();
            // X^T[k, t] = sum_t' X[t', k] I[t', t], 16 tokens at a time
            const uint32_t id_turn = make_idesc(64, 16, true, false);
            if (elect_one()) {
                if (PER_TOKEN) {
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        mma_ss(tm + U_WR + 16 * q, mnmaj(offsetof(MildSmem, in) + T_W * TILE_BYTES, q), kmaj(offsetof(MildSmem, ident), 0), id_turn, false);
                }
#pragma unroll
                for (int q = 0; q < 4; q++)
                    mma_ss(tm_hi + U_WR + 16 * q, mnmaj(offsetof(MildSmem, in) + T_R * TILE_BYTES, q), kmaj(offsetof(MildSmem, ident), 0), id_turn, false);
#pragma unroll
                for (int q = 0; q < 4; q++)
                    mma_ss(tm + U_KV + 16 * q, mnmaj(offsetof(MildSmem, in) + T_K * TILE_BYTES, q), kmaj(offsetof(MildSmem, ident), 0), id_turn, false);
                mma_commit(&s.turned);
            }
            stage = 1;
            if (!wait(&s.full[1], ph)) break;
            const uint32_t id_kk = make_idesc(64, 64, false, false), id_mm = make_idesc(64, 64, true, true),
                           id_km = make_idesc(64, 64, false, true);
            if (elect_one()) {
                // P[t,s] = sum_v gy[t,v] v[s,v]
#pragma unroll
                for (int q = 0; q < 4; q++)
                    mma_ss(tm_hi + U_AP, kmaj(offsetof(MildSmem, in) + T_GY * TILE_BYTES, q), kmaj(offsetof(MildSmem, in) + T_V * TILE_BYTES, q), id_kk, q > 0);
                // Gr[k,t] = sum_v S'[k,v] gy[t,v];  Gk[k,s] = sum_v D'[k,v] v[s,v]
#pragma unroll
                for (int q = 0; q < 4; q++)
                    mma_ss(tm + U_G, kmaj(offsetof(MildSmem, in) + T_S * TILE_BYTES, q), kmaj(offsetof(MildSmem, in) + T_GY * TILE_BYTES, q), id_kk, q > 0);
#pragma unroll
                for (int q = 0; q < 4; q++)
                    mma_ss(tm_hi + U_G, kmaj(offsetof(MildSmem, in) + T_D * TILE_BYTES, q), kmaj(offsetof(MildSmem, in) + T_V * TILE_BYTES, q), id_kk, q > 0);
                mma_commit(&s.early);
            }
            stage = 2;
            if (!wait(&s.ops, ph)) break;
            tc_fence_after();
            // A[t,s] = sum_k Rt[t,k] Kt[s,k]   (both tiles are [channel][token])
            if (elect_one()) {
#pragma unroll
                for (int q = 0; q < 4; q++)
                    mma_ss(tm + U_AP, mnmaj(offsetof(MildSmem, rt), q), mnmaj(offsetof(MildSmem, kt), q), id_mm, q > 0);
                mma_commit(&s.score);
                if (more) load0(x, ph ^ 1);
            }
            stage = 3;
            if (!wait(&s.mask, ph)) break;
            tc_fence_after();
            if (elect_one()) {
                // Gr[k,t] += sum_s Kt[s,k] P~[t,s];  Gk[k,s] += sum_t Rt[t,k] P~[t,s]
#pragma unroll
                for (int q = 0; q < 4; q++)
                    mma_ss(tm + U_G, kmaj(offsetof(MildSmem, kt), q), kmaj(offsetof(MildSmem, pt), q), id_kk, true);
#pragma unroll
                for (int q = 0; q < 4; q++)
                    mma_ss(tm_hi + U_G, kmaj(offsetof(MildSmem, rt), q), mnmaj(offsetof(MildSmem, pt), q), id_km, true);
                mma_commit(&s.grad);
                // gv[s,v] = sum_t A~[t,s] gy[t,v] + sum_k Kt[s,k] D'[k,v]
#pragma unroll
                for (int q = 0; q < 4; q++)
                    mma_ss(tm_hi + U_KV, mnmaj(offsetof(MildSmem, at), q), mnmaj(offsetof(MildSmem, in) + T_GY * TILE_BYTES, q), id_mm, q > 0);
#pragma unroll
                for (int q = 0; q < 4; q++)
                    mma_ss(tm_hi + U_KV, mnmaj(offsetof(MildSmem, kt), q), mnmaj(offsetof(MildSmem, in) + T_D * TILE_BYTES, q), id_mm, true);
                mma_commit(&s.gv);
                if (more) load1a(x);
            }
            stage = 4;
            if (!wait(&s.gv, ph)) break;
            if (more && elect_one()) load1b(x);
            all = true;
            if (!wait(&s.epi, ph)) break;
            tc_fence_after();
            stage = 5;
        } while (false);
        if (stage < 5) {
            fine = false;
            if (P.status && elect_one()) atomicOr(P.status, 4);
            // let whatever is in flight finish before shared and tensor memory go away
            if (loads) { mbar_wait(&s.full[0], ph, 200000u); mbar_wait(&s.full[1], ph, 200000u); }
            uint64_t *last[5] = {nullptr, &s.turned, &s.early, &s.score, &s.gv};
            for (int q = 1; q <= stage; q++) mbar_wait(last[q], ph, 200000u);
            if (more && stage >= 3) {
                // (those of the next chunk: the second group is short of two loads if the wait for gv ran out, and would
                // never complete)
                mbar_wait(&s.full[0], ph ^ 1, 200000u);
                if (stage == 4 && !all && elect_one()) load1b(x);
                if (stage == 4) mbar_wait(&s.full[1], ph ^ 1, 200000u);
            }
        }
        loads = more;
        chunk = next;
    }
    return fine;
}

// What the turned inputs should have been where an element of the chunk is infinite or NaN: it has met the identity's
// zeros and made the other 15 of its run NaN.  The thread's r and k and, summed up, its log2-decays (of `nv` valid tokens)
// go to their places in tensor memory (wr: w's), the decays' total to stot; returned: which decays are below the floor.
// (Out of line: written into the loop, where it never ran, it made the backward pass of a 7B segment 421 us instead of 407.)
template <bool PER_TOKEN>
__device__ __noinline__ unsigned mild_inputs_again(MildSmem &s, uint32_t wr, int k, int t0, int nv) {
    auto at = [&](const Tile &t, int i) {
        return __bfloat162float(*reinterpret_cast<const __nv_bfloat16 *>(t.b + tile_off(t0 + i, k >> 3) + 2 * (k & 7)));
    };
    unsigned dead = 0;
    float v[16];
    if (PER_TOKEN) {
        float sum = 0.f;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            bool live;
            const float l2 = log2_decay(at(s.in[T_W], i), WKV_W_RAW, live);
            if (!live) dead |= 1u << i;
            if (t0 + i < nv) sum += l2;
            v[i] = sum;
        }
        s.stot[t0 >> 4][k] = sum;
        tmem_st16_split32(wr, v);
    }
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = at(s.in[T_R], i);
    tmem_st16_split32(wr + (16u << 16), v);
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = at(s.in[T_K], i);
    tmem_st16_split32(wr + (U_KV - U_WR), v);
    tmem_st_wait();
    return dead;
}

// The compute warps of the same chunks; bar: their named barrier.
template <bool PER_TOKEN>
__device__ __forceinline__ bool
mild_compute(const CUtensorMap &map_gr, const CUtensorMap &map_gk, const CUtensorMap &map_gv, const CUtensorMap &map_gw,
             const BwdParams &P, MildSmem &s, const uint32_t tm, const int warp, const int bar, const int first, const int stride) {
    const int lane = threadIdx.x & 31, tid = 32 * warp + lane, n = P.nchunk;
    const uint32_t LIM = P.wait_limit;
    auto wait = [&](uint64_t *bar, uint32_t ph) {
        if (mbar_wait_or_abort(bar, ph, &s.abort_flag, LIM)) return true;
        *reinterpret_cast<volatile int *>(&s.abort_flag) = 1;
        return false;
    };
    ChunkWalk walk(P.mildflag, first, stride, P.total, 1u);
    int chunk = walk.next();
    if (chunk < 0) return true;
    const int wg = warp >> 2, w4 = warp & 3;
    const uint32_t lo_lanes = (uint32_t)(32 * w4), hi_lanes = lo_lanes + 16, tcol = 16 * wg;
    // a head's u, and a static decay, are fetched one chunk ahead (as they are in memory: a conversion would wait)
    auto head_at = [&](int c) {
        const int bh = P.by_n.div(c);
        return (bh - P.by_H.div(bh) * P.H) * 64 + 16 * w4 + (lane & 15);
    };
    __nv_bfloat16 u_next = P.u[head_at(chunk)];
    float x_next = PER_TOKEN ? 0.f : P.wvec[head_at(chunk)];
    if (wg == 0 && lane < 16) s.uf[0][16 * w4 + lane] = __bfloat162float(u_next);
    compute_sync(bar);
    bool fine = true;
    for (uint32_t ph = 0; chunk >= 0; ph ^= 1) {
        const int next = walk.next();
        // (what follows from the lane is computed again for every chunk: kept across the loop, the addresses alone would
        // not leave enough registers for the rest)
        int ln = lane;
        asm volatile("" : "+r"(ln));
        const int hh = ln >> 4, k = 16 * w4 + (ln & 15), t0 = 32 * hh + 16 * wg, run4 = 2 * hh + wg;  // the thread's channel and tokens
        const int bh = P.by_n.div(chunk), j = chunk - bh * n, b = P.by_H.div(bh), h = bh - b * P.H;
        const bool whole = (j + 1) * CH <= P.T;
        float lw = 0.f;
        bool live = true;
        if (!PER_TOKEN) lw = log2_decay(x_next, P.w_kind, live);
        {
            const int at = head_at(next >= 0 ? next : chunk);
            u_next = P.u[at];
            if (!PER_TOKEN) x_next = P.wvec[at];
        }

        // ------------------------------------------------ operand pass
        // first, while the inputs are being turned: the bonus term of the score diagonal, sum_k r_t u k_t, from the raw
        // tiles: a thread takes 16 channels of token k
        wait(&s.full[0], ph);
        bool odd;                 // an infinite or NaN r or k among those that the thread has seen
        {
            f2 d2 = both(0.f);
#pragma unroll
            for (int c = 0; c < 2; c++) {
                const int c8 = 2 * run4 + c;
                float a[8], d[8], uq[8];
                unpack8(ld_tile(s.in[T_R], k, c8), a);
                unpack8(ld_tile(s.in[T_K], k, c8), d);
                {
                    const float4 u0 = *reinterpret_cast<const float4 *>(s.uf[ph] + 8 * c8), u1 = *reinterpret_cast<const float4 *>(s.uf[ph] + 8 * c8 + 4);
                    uq[0] = u0.x; uq[1] = u0.y; uq[2] = u0.z; uq[3] = u0.w; uq[4] = u1.x; uq[5] = u1.y; uq[6] = u1.z; uq[7] = u1.w;
                }
#pragma unroll
                for (int q = 0; q < 8; q += 2)
                    d2 = fma2(mul2(make_float2(a[q], a[q + 1]), make_float2(uq[q], uq[q + 1])), make_float2(d[q], d[q + 1]), d2);
            }
            float diag = d2.x + d2.y;
            odd = !(fabsf(diag) <= FLT_MAX);
            diag += __shfl_xor_sync(0xffffffffu, diag, 16);
            if (hh == 0) s.dpart[wg][k] = diag;
        }
        unsigned dead = 0;        // tokens whose decay was below the floor
        float base;               // log2-decay summed up to before the thread's first token, less m
        uint32_t rtp[8], ktp[8];  // the thread's operands, two tokens a word: wanted again in the epilogue
        wait(&s.turned, ph);
        tc_fence_after();
        {
            float c[16], r[16];
            if (PER_TOKEN) {
                tmem_ld16_split32(tmem_addr(tm, lo_lanes, U_WR + tcol), c);
                tmem_ld_wait();
                float mx = 0.f;
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    c[i] = exp2f(fmaf(c[i], LOG2E, LOG2_LOG2E));        // minus the log2-decay
                    mx = fmaxf(mx, c[i]);
                }
                if (mx > -L2_FLOOR) {
#pragma unroll
                    for (int i = 0; i < 16; i++)
                        if (c[i] > -L2_FLOOR) { dead |= 1u << i; c[i] = -L2_FLOOR; }
                }
                if (!whole) {
#pragma unroll
                    for (int i = 0; i < 16; i++)
                        if (j * CH + t0 + i >= P.T) c[i] = 0.f;
                }
                c[0] = -c[0];
#pragma unroll
                for (int i = 1; i < 16; i++) c[i] = c[i - 1] - c[i];
                odd |= !(c[15] <= 0.f);
                // the four runs of 16 tokens of a channel meet
                s.stot[run4][k] = c[15];
            }
            // the outputs of the chunk before have left their tiles (read below by everyone's writes)
            if (tid == 0) tma_store_wait_read();
            if (compute_sync_or(odd, bar)) {
                dead = mild_inputs_again<PER_TOKEN>(s, tmem_addr(tm, lo_lanes, U_WR + tcol), k, t0, P.T - j * CH);
                if (PER_TOKEN) { tmem_ld16_split32(tmem_addr(tm, lo_lanes, U_WR + tcol), c); tmem_ld_wait(); }
                compute_sync(bar);
            }
            tmem_ld16_split32(tmem_addr(tm, hi_lanes, U_WR + tcol), r);
            const float m = rintf(s.cst[ph][0][k]);
            if (PER_TOKEN) {
                base = -m;
                if (hh) base += s.stot[0][k] + s.stot[1][k];
                if (wg) base += s.stot[hh ? 2 : 0][k];
            } else {
                const int nv = P.T - j * CH;
                base = (float)min(t0, nv) * lw - m;
#pragma unroll
                for (int i = 0; i < 16; i++) c[i] = (float)(min(t0 + i + 1, nv) - min(t0, nv)) * lw;
            }
            vadds<16>(c, c, base);
            tmem_ld_wait();
            float prev = base;
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
                const f2 o = mul2(make_float2(r[i], r[i + 1]), make_float2(exp2f(prev), exp2f(c[i])));
                prev = c[i + 1];
                rtp[i >> 1] = pack2(o.x, o.y);
            }
            st_tile(s.rt, k, (t0 >> 3), make_uint4(rtp[0], rtp[1], rtp[2], rtp[3]));
            st_tile(s.rt, k, (t0 >> 3) + 1, make_uint4(rtp[4], rtp[5], rtp[6], rtp[7]));
            tmem_ld16_split32(tmem_addr(tm, lo_lanes, U_KV + tcol), r);        // (k)
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
                const f2 o = mul2(make_float2(r[i], r[i + 1]), make_float2(exp2f(-c[i]), exp2f(-c[i + 1])));
                ktp[i >> 1] = pack2(o.x, o.y);
            }
            st_tile(s.kt, k, (t0 >> 3), make_uint4(ktp[0], ktp[1], ktp[2], ktp[3]));
            st_tile(s.kt, k, (t0 >> 3) + 1, make_uint4(ktp[4], ktp[5], ktp[6], ktp[7]));
            tmem_st16_split32(tmem_addr(tm, lo_lanes, U_WR + tcol), c);
            tmem_st_wait();
        }
        fence_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s.ops);

        // ------------------------------------------------ mask pass
        // lo lanes build A~ (row t), hi lanes build P~ (row t); this group's 32 columns
        const bool lo = hh == 0;
        const int row = k, col0 = 32 * wg;              // score row, first score column
        const bool diag_warp = (w4 >= 2) == (wg == 1), cross_warp = wg == 0 && w4 >= 2;
        wait(&s.early, ph);
        wait(&s.score, ph);
        tc_fence_after();
        {
            const int t = row;
            float a[32];
            if (diag_warp || cross_warp) {
                tmem_ld16(tmem_addr(tm, lo_lanes, U_AP + col0), a);
                tmem_ld16(tmem_addr(tm, lo_lanes, U_AP + col0 + 16), a + 16);
                tmem_ld_wait();
            }
            if (diag_warp) {
                // The 16 x 16 block on the diagonal: columns left of the row's own are kept, the diagonal is the bonus
                // term in A~, and zero in P~ with p_tt set aside.  Rows 0..15 of the 32 have it in columns 0..15 and
                // cannot reach columns 16..31, rows 16..31 keep all of columns 0..15.
                const int lim = ln & 15, at = w4 & 1 ? 16 : 0;
                if (!lo) {       // (p_tt is picked by way of gr's tile, which is free: cheaper than 16 selections)
                    float4 *p = reinterpret_cast<float4 *>(s.gr.b + t * 64);
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        p[q] = at ? make_float4(a[16 + 4 * q], a[17 + 4 * q], a[18 + 4 * q], a[19 + 4 * q])
                                  : make_float4(a[4 * q], a[4 * q + 1], a[4 * q + 2], a[4 * q + 3]);
                    s.ptt[t] = reinterpret_cast<const float *>(p)[lim];
                }
                if (at) {
#pragma unroll
                    for (int q = 0; q < 16; q++) a[16 + q] = q < lim ? a[16 + q] : 0.f;
                } else {
#pragma unroll
                    for (int q = 0; q < 16; q++) { a[q] = q < lim ? a[q] : 0.f; a[16 + q] = 0.f; }
                }
            } else if (!cross_warp) {   // upper-right block: nothing survives
#pragma unroll
                for (int q = 0; q < 32; q++) a[q] = 0.f;
            }
            Tile &dst = lo ? s.at : s.pt;
#pragma unroll
            for (int c8 = 0; c8 < 4; c8++) st_tile(dst, t, (col0 >> 3) + c8, pack8(a + 8 * c8));
            if (diag_warp && lo)
                *reinterpret_cast<__nv_bfloat16 *>(s.at.b + tile_off(t, t >> 3) + (t & 7) * 2) = __float2bfloat16_rn(s.dpart[0][t] + s.dpart[1][t]);
        }
        fence_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s.mask);

        // ------------------------------------------------ epilogue
        int ke = k;
        asm volatile("" : "+r"(ke));
        const int c8k = ke >> 3, b0 = t0 * TILE_ROW_BYTES + (ke & 7) * 2;
        // values of the thread's channel at its tokens i and i + 1
        auto put2 = [&](Tile &o, int i, const f2 &v) {
            const uint32_t p = pack2(v.x, v.y);
            *reinterpret_cast<unsigned short *>(o.b + b0 + i * TILE_ROW_BYTES + ((c8k ^ (i & 7)) << 4)) = (unsigned short)p;
            *reinterpret_cast<unsigned short *>(o.b + b0 + (i + 1) * TILE_ROW_BYTES + ((c8k ^ ((i + 1) & 7)) << 4)) = (unsigned short)(p >> 16);
        };
        wait(&s.mask, ph);         // (every warp's share of ptt)
        wait(&s.grad, ph);
        tc_fence_after();
        // The decay gradient of token t is  glw_t = K_j + sum_{t'<=t} (a_t' + b_t') - b_t, times the token's log-decay
        float glw[16], run = 0.f;
        {
            f2 gus = both(0.f);
            float prev = base;
            const float u = s.uf[ph][k];
#pragma unroll
            for (int qt = 0; qt < 4; qt++) {        // (four tokens at a time: registers)
                float Gr[4], Gk[4], r[4], kk[4], c[4];
                tmem_ld4_split32(tmem_addr(tm, lo_lanes, U_G + tcol + 4 * qt), Gr);
                tmem_ld4_split32(tmem_addr(tm, hi_lanes, U_G + tcol + 4 * qt), Gk);
                tmem_ld4_split32(tmem_addr(tm, lo_lanes, U_WR + tcol + 4 * qt), c);
                tmem_ld4_split32(tmem_addr(tm, hi_lanes, U_WR + tcol + 4 * qt), r);
                tmem_ld4_split32(tmem_addr(tm, lo_lanes, U_KV + tcol + 4 * qt), kk);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 4; i += 2) {
                    const f2 gr2 = make_float2(Gr[i], Gr[i + 1]), gk2 = make_float2(Gk[i], Gk[i + 1]),
                             r2 = make_float2(r[i], r[i + 1]), k2 = make_float2(kk[i], kk[i + 1]),
                             p2 = *reinterpret_cast<const f2 *>(s.ptt + t0 + 4 * qt + i);
                    const f2 fr = make_float2(exp2f(prev), exp2f(c[i])), fk = make_float2(exp2f(-c[i]), exp2f(-c[i + 1]));
                    // (below, c: the tokens' own log-decays)
                    const float l = c[i] - prev;
                    prev = c[i + 1];
                    c[i + 1] -= c[i];
                    c[i] = l;
                    const f2 pr = mul2(p2, r2), pk = mul2(p2, k2);
                    gus = fma2(pr, k2, gus);
                    put2(s.gr, 4 * qt + i, fma2(pk, both(u), mul2(fr, gr2)));
                    put2(s.gk, 4 * qt + i, fma2(pr, both(u), mul2(fk, gk2)));
                    const f2 a2 = mul2(unpack2(rtp[2 * qt + (i >> 1)] ^ 0x80008000u), gr2);
                    const f2 z = fma2(unpack2(ktp[2 * qt + (i >> 1)]), gk2, a2);
                    glw[4 * qt + i] = run + a2.x;
                    run += z.x;
                    glw[4 * qt + i + 1] = run + a2.y;
                    run += z.y;
                }
                // (kept in A's place: the registers are needed)
                if (PER_TOKEN) tmem_st4_split32(tmem_addr(tm, lo_lanes, U_AP + tcol + 4 * qt), c);
            }
            s.rtot[run4][k] = run;
            s.gup[run4][k] = gus.x + gus.y;
        }
        // the accumulators and the turned inputs have been read: the next chunk may have their place
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s.epi);
        wait(&s.gv, ph);
        tc_fence_after();
        {
            // gv: accumulator [token 16 w4 + l16][value 32 hh + 16 wg ..]; A~ has been read
            float gv[16];
            tmem_ld16_split32(tmem_addr(tm, hi_lanes, U_KV + tcol), gv);
            tmem_ld_wait();
            st_tile(s.at, row, (t0 >> 3), pack8(gv));
            st_tile(s.at, row, (t0 >> 3) + 1, pack8(gv + 8));
        }
        compute_sync(bar);
        {
            float g0 = s.cst[ph][1][k];           // the constant of the chunk start plus the earlier runs' totals
            if (hh) g0 += s.rtot[0][k] + s.rtot[1][k];
            if (wg) g0 += s.rtot[hh ? 2 : 0][k];
            if (PER_TOKEN) {
                // times the floored log-decay of the token, zero where the floor was hit (no gradient)
                float l2[16];
                tmem_ld16_split32(tmem_addr(tm, lo_lanes, U_AP + tcol), l2);
                tmem_ld_wait();
                vadds<16>(glw, glw, g0);
                if (dead) {
#pragma unroll
                    for (int i = 0; i < 16; i++)
                        if (dead >> i & 1) glw[i] = 0.f;
                }
#pragma unroll
                for (int i = 0; i < 16; i += 2)
                    put2(s.pt, i, mul2(mul2(make_float2(glw[i], glw[i + 1]), both(LN2)), make_float2(l2[i], l2[i + 1])));
            } else {
                float tot = 0.f;
#pragma unroll
                for (int i = 0; i < 16; i++)
                    if (j * CH + t0 + i < P.T) tot += g0 + glw[i];
                s.gwp[run4][k] = tot;
            }
        }
        if (run4 == 0) s.uf[ph ^ 1][k] = __bfloat162float(u_next);
        fence_async_smem();
        tc_fence_before();
        fine = !compute_sync_or(*reinterpret_cast<volatile int *>(&s.abort_flag) != 0, bar);
        if (!fine) break;
        if (tid == 0) {
            tma_store_3d(&map_gr, &s.gr, h * 64, j * CH, b);
            tma_store_3d(&map_gk, &s.gk, h * 64, j * CH, b);
            tma_store_3d(&map_gv, &s.at, h * 64, j * CH, b);
            if (PER_TOKEN) tma_store_3d(&map_gw, &s.pt, h * 64, j * CH, b);
            tma_store_commit();
        }
        // per-chunk partials, folded later in a fixed order
        if (wg == 1 && hh == 0)
            P.gu_part[(size_t)chunk * 64 + k] = (s.gup[0][k] + s.gup[1][k]) + (s.gup[2][k] + s.gup[3][k]);
        else if (!PER_TOKEN && wg == 1)
            P.gw_part[(size_t)chunk * 64 + k] = live ? ((s.gwp[0][k] + s.gwp[1][k]) + (s.gwp[2][k] + s.gwp[3][k])) * (lw * LN2) : 0.f;
        chunk = next;
    }
    if (tid == 0) {
        tma_store_wait_read();   // the tiles must outlive the reads of the bulk stores
        if (!fine && P.status) atomicOr(P.status, 4);
    }
    return fine;
}

#define BWD_MAPS                                                                                              \
    const __grid_constant__ CUtensorMap map_r, const __grid_constant__ CUtensorMap map_k,                    \
        const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_w,                \
        const __grid_constant__ CUtensorMap map_gy, const __grid_constant__ CUtensorMap map_s,               \
        const __grid_constant__ CUtensorMap map_d, const __grid_constant__ CUtensorMap map_gr,               \
        const __grid_constant__ CUtensorMap map_gk, const __grid_constant__ CUtensorMap map_gv,              \
        const __grid_constant__ CUtensorMap map_gw

// One CTA per SM, two groups in it that share nothing but the tensor memory's allocation: eight compute warps, a feeder warp
// and half of the shared memory each.  Registers: the compute warps take what the feeders' warpgroup gives up (512 x 112
// + 128 x 32 = 640 x 96); as two CTAs of nine warps they would have 96, and spill in every chunk.  The flag that the
// forward kernel left for a chunk says which body it takes: a group does its mild chunks (all chunks of ordinary
// data), then its steep ones.
constexpr int BWD_GROUPS = 2, BWD_THREADS = 640;      // warps 0..15 compute, 16 and 17 feed, 18 and 19 only fill a warpgroup
template <bool PER_TOKEN>
__global__ void __launch_bounds__(BWD_THREADS, 1) k_chunk_bwd(BWD_MAPS, const BwdParams P) {
    pdl_wait();
    pdl_trigger();
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31;
    const int warp_id = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);   // tells the compiler it is uniform across the warp
    const bool feeder = warp_id >= 16;
    const int grp = feeder ? warp_id & 1 : warp_id >> 3, warp = warp_id & 7;
    unsigned char *mem = smem_raw + grp * BWD_SMEM;
    MildSmem &s = *reinterpret_cast<MildSmem *>(mem);
    // (behind both groups' memory, of which each makes another use once its mild chunks are done)
    uint32_t *tmem_base = reinterpret_cast<uint32_t *>(smem_raw + BWD_GROUPS * BWD_SMEM);

    // the swizzled tiles need a 1024-byte aligned base; refuse to run otherwise
    if ((smem_u32(smem_raw) & 1023u) != 0) {
        if (threadIdx.x == 0 && P.status) atomicOr(P.status, 8);
        return;
    }
    if ((warp_id == 16 || warp_id == 17) && lane == 0) {
        mbar_init(&s.full[0], 1); mbar_init(&s.full[1], 1);
        mbar_init(&s.turned, 1); mbar_init(&s.early, 1); mbar_init(&s.score, 1); mbar_init(&s.grad, 1); mbar_init(&s.gv, 1);
        mbar_init(&s.ops, 8); mbar_init(&s.mask, 8); mbar_init(&s.epi, 8);
        s.abort_flag = 0;
        fence_mbar_init();
    }
    if (!feeder && warp == 7) {
        const int row = lane >> 1, c8 = lane & 1, one = row - 8 * c8;
        const uint32_t v = 0x3F80u << (16 * (one & 1));
        *reinterpret_cast<uint4 *>(s.ident + tile_off(row, c8)) =
            make_uint4(one >> 1 == 0 ? v : 0u, one >> 1 == 1 ? v : 0u, one >> 1 == 2 ? v : 0u, one >> 1 == 3 ? v : 0u);
        fence_async_smem();
    }
    if (warp_id == 0) { tmem_alloc(tmem_base, BWD_TMEM_COLS * BWD_GROUPS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm0 = __shfl_sync(0xffffffffu, *tmem_base, 0), tm = tm0 + BWD_TMEM_COLS * grp;
    // (the CTAs' first groups come first: a call of few chunks has an SM for each, and so has a last round of few)
    const int first = grp * (int)gridDim.x + (int)blockIdx.x, stride = (int)gridDim.x * BWD_GROUPS;
    const int bar = 1 + grp, bar_all = 1 + BWD_GROUPS + grp;     // named barriers: of the compute warps, of the whole group
    if (feeder) {
        regs_give_up<32>();
        if (warp_id < 18) {
            const bool fine = mild_feed<PER_TOKEN>(map_r, map_k, map_v, map_w, map_gy, map_s, map_d, P, s, tm, first, stride);
            compute_sync_or(!fine, bar_all, 288);
        }
    } else {
        regs_take<112>();
        const bool fine = mild_compute<PER_TOKEN>(map_gr, map_gk, map_gv, map_gw, P, s, tm, warp, bar, first, stride);
        tc_fence_before();
        // (no thread goes on where one has given up)
        if (!compute_sync_or(!fine, bar_all, 288)) {
            tc_fence_after();
            ChunkWalk walk(P.mildflag, first, stride, P.total, 0u);
            int chunk = walk.next();
            if (chunk >= 0) {
                SteepSmem &q = *reinterpret_cast<SteepSmem *>(mem);
                const int n = P.nchunk, tid = 32 * warp + lane;
                if (tid == 0) {
                    uint64_t *old[10] = {&s.full[0], &s.full[1], &s.turned, &s.early, &s.ops, &s.score, &s.mask, &s.grad, &s.gv, &s.epi};
                    for (int i = 0; i < 10; i++) mbar_inval(old[i]);
                    mbar_init(&q.load_bar, 1);
                    // lane 0 of every compute warp commits to every barrier, whether or not it issued a share of the group
                    mbar_init(&q.bar_early, 8); mbar_init(&q.bar_score, 8); mbar_init(&q.bar_grad, 8); mbar_init(&q.bar_gv, 8);
                    fence_mbar_init();
                }
                compute_sync(bar);
                for (uint32_t ph = 0; chunk >= 0; ph ^= 1) {
                    const int bh = P.by_n.div(chunk), j = chunk - bh * n, b = P.by_H.div(bh), h = bh - b * P.H;
                    const int next = walk.next();
                    if (tid == 32 && next >= 0) {       // the next chunk's tiles come from L2
                        const int bh2 = P.by_n.div(next), j2 = next - bh2 * n, b2 = P.by_H.div(bh2), h2 = bh2 - b2 * P.H;
                        tma_prefetch_l2_3d(&map_r, h2 * 64, j2 * CH, b2);
                        tma_prefetch_l2_3d(&map_k, h2 * 64, j2 * CH, b2);
                        tma_prefetch_l2_3d(&map_v, h2 * 64, j2 * CH, b2);
                        if (PER_TOKEN) tma_prefetch_l2_3d(&map_w, h2 * 64, j2 * CH, b2);
                        tma_prefetch_l2_3d(&map_gy, h2 * 64, j2 * CH, b2);
                        tma_prefetch_l2_3d(&map_s, 0, 0, bh2 * (n + 1) + j2);
                        tma_prefetch_l2_3d(&map_d, 0, 0, bh2 * (n + 1) + j2 + 1);
                    }
                    if (tid == 0 && j != P.skip_load) {
                        mbar_expect_tx(&q.load_bar, (PER_TOKEN ? 7 : 6) * TILE_BYTES);
                        tma_load_3d(&q.in[T_R], &map_r, &q.load_bar, h * 64, j * CH, b);
                        tma_load_3d(&q.in[T_K], &map_k, &q.load_bar, h * 64, j * CH, b);
                        tma_load_3d(&q.in[T_V], &map_v, &q.load_bar, h * 64, j * CH, b);
                        if (PER_TOKEN) tma_load_3d(&q.in[T_W], &map_w, &q.load_bar, h * 64, j * CH, b);
                        tma_load_3d(&q.in[T_GY], &map_gy, &q.load_bar, h * 64, j * CH, b);
                        tma_load_3d(&q.in[T_S], &map_s, &q.load_bar, 0, 0, bh * (n + 1) + j);
                        tma_load_3d(&q.in[T_D], &map_d, &q.load_bar, 0, 0, bh * (n + 1) + j + 1);
                    }
                    if (tid >= 128 && tid < 128 + CH) q.uf[tid - 128] = __bfloat162float(P.u[h * 64 + tid - 128]);
                    compute_sync(bar);
                    tc_fence_after();
                    if (!bwd_steep<PER_TOKEN>(map_gr, map_gk, map_gv, map_gw, P, q, tm, warp, bar, chunk, ph)) break;
                    tc_fence_before();
                    compute_sync(bar);      // the tiles are free: the stores have read theirs
                    chunk = next;
                }
            }
        }
        tc_fence_before();
    }
    __syncthreads();
    if (warp_id == 0) tmem_dealloc(tm0, BWD_TMEM_COLS * BWD_GROUPS);
}

// sum the per-chunk partials: out[bh*64 + k] = sum_j part[(bh*n + j)*64 + k]
__global__ void k_reduce_partials(const float *__restrict__ part, float *__restrict__ out, int n, int total) {
    pdl_wait();
    pdl_trigger();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int bh = i >> 6, k = i & 63;
    float acc = 0.f;
    for (int j = 0; j < n; j++) acc += part[((size_t)bh * n + j) * 64 + k];
    out[i] = acc;
}

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

struct BwdLayout {
    size_t status, sck, dck, e0, gu_part, gw_part, groups, wconv, total;
};
BwdLayout bwd_layout(const wkv_args_t *a, bool per_token_w) {
    const size_t n = (a->T + CH - 1) / CH, bh = (size_t)a->B * a->H;
    const GroupPlan gp = plan_groups((int)bh, (int)n, a->time_groups);
    BwdLayout L;
    L.status = 0;
    L.sck = 256;
    L.dck = L.sck + align256(ckpt_layout(a->B, a->T, a->H).total);
    L.e0 = L.dck + align256(bh * (n + 1) * 64 * 64 * 2);
    L.gu_part = L.e0 + align256(bh * (n + 1) * 64 * 4);
    L.gw_part = L.gu_part + align256(bh * n * 64 * 4);
    L.groups = L.gw_part + (per_token_w ? 0 : align256(bh * n * 64 * 4));
    // one region serves the forward re-run (when no hand-over was given) and then the dS scan
    L.wconv = L.groups + (gp.G > 1 ? group_layout(bh * gp.G).total : 0);
    L.total = L.wconv + chunked_wconv_bytes(a, per_token_w);
    return L;
}

}  // namespace

size_t chunked_backward_workspace(const wkv_args_t *a, bool per_token_w) { return bwd_layout(a, per_token_w).total; }

int chunked_backward(const wkv_args_t *a0, bool per_token_w, const CallOpts &opt, cudaStream_t stream) {
    wkv_args_t args = *a0;
    wkv_args_t *a = &args;
    const int B = a->B, T = a->T, H = a->H, C = H * 64, n = (T + CH - 1) / CH, BH = B * H;
    const BwdLayout L = bwd_layout(a, per_token_w);
    char *ws = (char *)a->workspace;
    int *status = opt.status ? opt.status : (int *)ws;
    if (!opt.status && cudaMemsetAsync(ws, 0, 256, stream) != cudaSuccess) return WKV_ERR_LAUNCH;
    if (chunked_convert_w(a, per_token_w, ws + L.wconv, stream) != WKV_OK) return WKV_ERR_LAUNCH;
    // what the forward kernel leaves for this call: chunk-start states, r e^{cp}, chunk decays
    char *fwd_ck = a->state_ckpt ? (char *)a->state_ckpt : ws + L.sck;
    const CkptLayout CL = ckpt_layout(B, T, H);
    void *sck = fwd_ck + CL.sck, *dck = ws + L.dck;
    float *gu_part = (float *)(ws + L.gu_part), *gw_part = (float *)(ws + L.gw_part), *e0 = (float *)(ws + L.e0);

    // 1. chunk-start states (unless the forward call handed them over)
    if (!a->state_ckpt) {
        wkv_args_t f = *a;
        f.y = nullptr;
        f.state_out = nullptr;
        f.group_states = nullptr;
        f.group_states_mode = WKV_GROUP_STATES_NONE;
        const int err = chunked_forward_impl(&f, per_token_w, fwd_ck, ws + L.groups, opt, stream);
        if (err != WKV_OK) return err;
    }
    CUtensorMap mr, mk, mv, mw, mgy, ms, md, mgr, mgk, mgv, mgw, mrh;
    bool ok = make_btc_map(&mr, a->r, B, T, C) && make_btc_map(&mk, a->k, B, T, C) &&
              make_btc_map(&mv, a->v, B, T, C) && make_btc_map(&mgy, a->gy, B, T, C) &&
              make_btc_map(&mgr, a->gr, B, T, C) && make_btc_map(&mgk, a->gk, B, T, C) &&
              make_btc_map(&mgv, a->gv, B, T, C) && make_btc_map(&ms, sck, BH * (n + 1), 64, 64) &&
              make_btc_map(&md, dck, BH * (n + 1), 64, 64) && make_btc_map(&mrh, fwd_ck + CL.rhat, B, T, C);
    if (per_token_w) ok = ok && make_btc_map(&mw, a->w, B, T, C) && make_btc_map(&mgw, a->gw, B, T, C);
    else { mw = mr; mgw = mgr; }
    if (!ok) return WKV_ERR_LAUNCH;

    // 2. dS scan (with time groups: summary pass, group scan, full pass)
    {
        const GroupPlan gp = plan_groups(BH, n, a->time_groups);
        const GroupLayout GL = group_layout((size_t)BH * gp.G);
        char *g = ws + L.groups;
        DscanParams p;
        p.T = T; p.H = H; p.nchunk = n; p.layout = a->state_layout;
        p.G = gp.G; p.L = gp.L;
        p.dchunk = (const float *)(fwd_ck + CL.dchunk);
        p.dck = (__nv_bfloat16 *)dck; p.e0 = e0; p.status = status;
        p.wait_limit = opt.wait_limit;
        p.skip_load = opt.kernel == 1 ? opt.skip_load : -1;
        const size_t smem = sizeof(DscanSmem) + 1024;
        static unsigned char attr_done[64];
        if (!set_max_smem_once(k_chunk_dscan, (int)smem, attr_done)) return WKV_ERR_LAUNCH;
        if (gp.G > 1) {
            p.summary = 1;
            p.gstate_out = nullptr; p.gstart = nullptr; p.gstate_in = nullptr; p.fold = 0;
            p.gU = (float *)(g + GL.gU); p.gD = (float *)(g + GL.gD);
            if (launch_chained(k_chunk_dscan, dim3(BH * (gp.G - 1)), dim3(160), smem, stream, mrh, mgy, ms, p) != WKV_OK)
                return WKV_ERR_LAUNCH;
            if (gp.G > GROUP_FOLD_MAX &&
                launch_group_scan(g, BH, gp.G, a->gstate_out, a->state_layout, true, stream) != WKV_OK)
                return WKV_ERR_LAUNCH;
        }
        p.summary = 0;
        p.gstart = gp.G > GROUP_FOLD_MAX ? (const float *)(g + GL.gstart) : nullptr;
        p.gstate_out = p.gstart ? nullptr : a->gstate_out;
        p.fold = gp.G > 1 && gp.G <= GROUP_FOLD_MAX;
        p.gstate_in = a->gstate_in;
        if (!p.fold) { p.gU = nullptr; p.gD = nullptr; }
        if (launch_chained(k_chunk_dscan, dim3(BH * gp.G), dim3(160), smem, stream, mrh, mgy, ms, p) != WKV_OK)
            return WKV_ERR_LAUNCH;
    }
    // 3. per-chunk gradients
    {
        BwdParams p;
        p.T = T; p.H = H; p.nchunk = n; p.w_kind = a->w_kind;
        p.total = BH * n;
        p.by_n = FastDiv(n); p.by_H = FastDiv(H);
        p.u = (const __nv_bfloat16 *)a->u;
        p.wvec = per_token_w ? nullptr : (const float *)a->w;
        p.dchunk = (const float *)(fwd_ck + CL.dchunk);
        p.e0 = e0; p.gu_part = gu_part; p.gw_part = gw_part; p.status = status;
        p.wait_limit = opt.wait_limit;
        p.skip_load = opt.kernel == 2 ? opt.skip_load : -1;
        p.mildflag = (const unsigned char *)(fwd_ck + CL.mild);
        const size_t smem = BWD_SMEM * BWD_GROUPS + 16;     // (and the tensor memory's address)
        auto kern = per_token_w ? k_chunk_bwd<true> : k_chunk_bwd<false>;
        static unsigned char attr_done[2][64];
        if (!set_max_smem_once(kern, (int)smem, attr_done[per_token_w ? 1 : 0])) return WKV_ERR_LAUNCH;
        if (launch_chained(kern, dim3(std::min(p.total, device_sm_count())), dim3(BWD_THREADS), smem, stream, mr, mk, mv, mw, mgy, ms, md, mgr,
                           mgk, mgv, mgw, p) != WKV_OK)
            return WKV_ERR_LAUNCH;
    }
    // 4. fold the per-chunk partial sums: over the chunks and the batch, or over the chunks alone
    if (opt.gu_sum) {
        if (fold_param_grads(gu_part, per_token_w ? nullptr : gw_part, B, H, n, opt, stream) != WKV_OK) return WKV_ERR_LAUNCH;
    } else {
        const int total = BH * 64;
        if (launch_chained(k_reduce_partials, dim3((total + 255) / 256), dim3(256), 0, stream, (const float *)gu_part,
                           (float *)a->gu, n, total) != WKV_OK)
            return WKV_ERR_LAUNCH;
        if (!per_token_w && launch_chained(k_reduce_partials, dim3((total + 255) / 256), dim3(256), 0, stream,
                                           (const float *)gw_part, (float *)a->gw, n, total) != WKV_OK)
            return WKV_ERR_LAUNCH;
    }
    return WKV_OK;
}

}  // namespace wkv
