// Host-side creation of TMA tensor maps for [B, T, C] activation tensors.
// The driver entry point is looked up through the runtime, so the library does
// not link against libcuda.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace wkv {

typedef CUresult (*encode_tiled_fn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                    const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                    const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                    CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline encode_tiled_fn tensor_map_encoder() {
    static encode_tiled_fn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (encode_tiled_fn)p;
    }
    return fn;
}

// Map over a contiguous bf16 tensor [B, T, C]; box = 64 channels x 64 tokens x 1 batch row,
// 128-byte swizzle, out-of-range tokens read as zero.  A map depends on the base address and the shape only, so maps are
// remembered per host thread, in a direct-mapped table: a program that goes through the same buffers every step encodes
// each map once.  (A forward and backward call takes 16 maps and a training step goes through several segments' buffers:
// a list of the last 64, searched from its start, missed every time from five segments on.)
inline bool make_btc_map(CUtensorMap *map, const void *base, int B, int T, int C) {
    struct Entry {
        CUtensorMap map;
        const void *base;
        int B, T, C;
    };
    constexpr int LOG_SLOTS = 9;
    static thread_local Entry cache[1 << LOG_SLOTS];
    const uint64_t key = (uint64_t)(uintptr_t)base ^ (uint64_t)T << 40 ^ (uint64_t)C << 52 ^ (uint64_t)B << 48;
    Entry &e = cache[(key >> 8) * 0x9E3779B97F4A7C15ull >> (64 - LOG_SLOTS)];
    if (e.base == base && e.B == B && e.T == T && e.C == C && base != nullptr) {
        *map = e.map;
        return true;
    }
    encode_tiled_fn enc = tensor_map_encoder();
    if (!enc) return false;
    cuuint64_t dims[3] = {(cuuint64_t)C, (cuuint64_t)T, (cuuint64_t)B};
    cuuint64_t strides[2] = {(cuuint64_t)C * 2, (cuuint64_t)T * C * 2};
    cuuint32_t box[3] = {64, 64, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    const auto encode = [&] {
        return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void *>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    };
    if (encode() != CUDA_SUCCESS) {
        // a driver call, and the calling thread may not have been in the runtime yet (an autograd thread whose buffers all
        // came out of the allocator's cache): setting the device binds its context to the thread
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaSetDevice(dev) != cudaSuccess || encode() != CUDA_SUCCESS) return false;
    }
    e.base = base; e.B = B; e.T = T; e.C = C; e.map = *map;
    return true;
}

}  // namespace wkv
