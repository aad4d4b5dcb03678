// What the two v4 kernel files share: the decay parameter and the base-2 exponents.
#pragma once
#include "wkv_common.cuh"

namespace wkv {

constexpr float V4_MIN_VALUE = -1e38f;      // the exponent of an empty state
constexpr float V4_LOG2E = 1.4426950408889634f, V4_LN2 = 0.6931471805599453f;

// An empty state's exponent stays what it is in either base.
__device__ __forceinline__ float to_base2(float o) { return o <= V4_MIN_VALUE ? V4_MIN_VALUE : o * V4_LOG2E; }
__device__ __forceinline__ float from_base2(float o) { return o <= V4_MIN_VALUE ? V4_MIN_VALUE : o * V4_LN2; }

// w = -exp(time_decay): given as such (fp32), or as time_decay in one of the element types
struct Decay4 {
    const void *p;
    int raw_dtype;      // -1: p is w itself
    __device__ __forceinline__ float at(int c) const {
        if (raw_dtype < 0) return ((const float *)p)[c];
        const float x = raw_dtype == WKV_F32    ? ((const float *)p)[c]
                        : raw_dtype == WKV_BF16 ? __bfloat162float(((const __nv_bfloat16 *)p)[c])
                                                : __half2float(((const __half *)p)[c]);
        return -expf(x);
    }
};

}  // namespace wkv
