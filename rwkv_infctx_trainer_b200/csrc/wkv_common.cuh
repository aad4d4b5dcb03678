// Shared helpers of the WKV kernels: element-type traits and argument checks.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <initializer_list>
#include <utility>

#include "../../include/wkv_b200.h"

namespace wkv {

constexpr int HEAD = 64;  // head size N compiled in (RWKV-v6/src/model.py:313)

template <typename F> struct Elem;
template <> struct Elem<float> {
    static __device__ __forceinline__ float ld(const float *p) { return *p; }
    static __device__ __forceinline__ void st(float *p, float x) { *p = x; }
};
template <> struct Elem<__nv_bfloat16> {
    static __device__ __forceinline__ float ld(const __nv_bfloat16 *p) { return __bfloat162float(*p); }
    static __device__ __forceinline__ void st(__nv_bfloat16 *p, float x) { *p = __float2bfloat16_rn(x); }
};
template <> struct Elem<__half> {
    static __device__ __forceinline__ float ld(const __half *p) { return __half2float(*p); }
    static __device__ __forceinline__ void st(__half *p, float x) { *p = __float2half_rn(x); }
};

// ---- bf16 values in 32-bit words, element types chosen at run time, sums over a warp
__device__ __forceinline__ void unpack8(const uint4 &q, float *f) {
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        f[2 * i] = __uint_as_float(w[i] << 16);
        f[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
    }
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t *>(&h);
}
__device__ __forceinline__ uint4 pack8(const float *f) {
    return make_uint4(pack2(f[0], f[1]), pack2(f[2], f[3]), pack2(f[4], f[5]), pack2(f[6], f[7]));
}
__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
__device__ __forceinline__ void store_as(void *p, int dtype, size_t i, float x) {
    if (dtype == WKV_F32) ((float *)p)[i] = x;
    else if (dtype == WKV_BF16) ((__nv_bfloat16 *)p)[i] = __float2bfloat16_rn(x);
    else ((__half *)p)[i] = __float2half_rn(x);
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float sigmoidf(float x) { return __fdividef(1.f, 1.f + __expf(-x)); }

// Two fp32 values per instruction (fma.f32x2): half the issue slots of the scalar forms, same rounding.
typedef float2 f2;
__device__ __forceinline__ unsigned long long bits(const f2 &a) { return *reinterpret_cast<const unsigned long long *>(&a); }
__device__ __forceinline__ f2 from_bits(unsigned long long v) { return *reinterpret_cast<f2 *>(&v); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    unsigned long long r;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(bits(a)), "l"(bits(b)), "l"(bits(c)));
    return from_bits(r);
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    unsigned long long r;
    asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(bits(a)), "l"(bits(b)));
    return from_bits(r);
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    unsigned long long r;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(bits(a)), "l"(bits(b)));
    return from_bits(r);
}
__device__ __forceinline__ f2 unpack2(uint32_t q) { return make_float2(__uint_as_float(q << 16), __uint_as_float(q & 0xFFFF0000u)); }
__device__ __forceinline__ f2 both(float x) { return make_float2(x, x); }
__device__ __forceinline__ f2 sub2(f2 a, f2 b) { return fma2(b, both(-1.f), a); }
__device__ __forceinline__ f2 neg2(f2 a) { return make_float2(-a.x, -a.y); }
// the same on arrays, N even
template <int N>
__device__ __forceinline__ void vmul(float *o, const float *a, const float *b) {
#pragma unroll
    for (int i = 0; i < N; i += 2) {
        const f2 r = mul2(make_float2(a[i], a[i + 1]), make_float2(b[i], b[i + 1]));
        o[i] = r.x; o[i + 1] = r.y;
    }
}
template <int N>
__device__ __forceinline__ void vadd(float *o, const float *a, const float *b) {
#pragma unroll
    for (int i = 0; i < N; i += 2) {
        const f2 r = add2(make_float2(a[i], a[i + 1]), make_float2(b[i], b[i + 1]));
        o[i] = r.x; o[i + 1] = r.y;
    }
}
template <int N>
__device__ __forceinline__ void vsub(float *o, const float *a, const float *b) {
#pragma unroll
    for (int i = 0; i < N; i += 2) {
        const f2 r = sub2(make_float2(a[i], a[i + 1]), make_float2(b[i], b[i + 1]));
        o[i] = r.x; o[i + 1] = r.y;
    }
}
template <int N>
__device__ __forceinline__ void vfma(float *o, const float *a, const float *b, const float *c) {
#pragma unroll
    for (int i = 0; i < N; i += 2) {
        const f2 r = fma2(make_float2(a[i], a[i + 1]), make_float2(b[i], b[i + 1]), make_float2(c[i], c[i + 1]));
        o[i] = r.x; o[i + 1] = r.y;
    }
}
// o = a + s
template <int N>
__device__ __forceinline__ void vadds(float *o, const float *a, float s) {
#pragma unroll
    for (int i = 0; i < N; i += 2) {
        const f2 r = add2(make_float2(a[i], a[i + 1]), both(s));
        o[i] = r.x; o[i + 1] = r.y;
    }
}
// o = s * a + c
template <int N>
__device__ __forceinline__ void vaxpy(float *o, float s, const float *a, const float *c) {
#pragma unroll
    for (int i = 0; i < N; i += 2) {
        const f2 r = fma2(both(s), make_float2(a[i], a[i + 1]), make_float2(c[i], c[i + 1]));
        o[i] = r.x; o[i + 1] = r.y;
    }
}

inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
inline bool all_aligned(std::initializer_list<const void *> ps) {      // (NULL counts as aligned)
    for (const void *p : ps)
        if (!aligned16(p)) return false;
    return true;
}

// Programmatic dependent launch.  A kernel launched through launch_chained() may be scheduled
// while the kernel before it in the stream is still running, which hides its launch latency
// behind that kernel's last CTAs.  pdl_wait() returns once every earlier kernel of the stream
// has finished and its writes are visible: it is the first statement of every kernel launched
// this way, in every thread, before anything touches global memory -- and before any tensor
// memory is allocated, so that a waiting CTA never holds what a CTA of the earlier kernel still
// needs.  pdl_trigger() lets the next kernel be scheduled once every CTA of this one has called
// it or left.  Both are no-ops in an ordinary launch.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

inline std::atomic<unsigned long long> launch_count{0};     // launches of this process

// early: whether the kernel may be scheduled before the one in front of it has finished
template <typename... KArgs, typename... Args>
inline int launch_kernel(bool early, void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                          Args &&...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = early ? 1 : 0;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    launch_count.fetch_add(1, std::memory_order_relaxed);
    return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...) == cudaSuccess ? WKV_OK : WKV_ERR_LAUNCH;
}
template <typename... KArgs, typename... Args>
inline int launch_chained(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                          Args &&...args) {
    return launch_kernel(true, kern, grid, block, smem, stream, std::forward<Args>(args)...);
}

// cudaFuncAttributeMaxDynamicSharedMemorySize is a per-device property of a kernel: set it on
// the first launch on each device only (`done` is the call site's own per-device record)
template <class K>
inline bool set_max_smem_once(K kern, int bytes, unsigned char (&done)[64]) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    if (dev >= 0 && dev < 64 && __atomic_load_n(&done[dev], __ATOMIC_ACQUIRE)) return true;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return false;
    if (dev >= 0 && dev < 64) __atomic_store_n(&done[dev], (unsigned char)1, __ATOMIC_RELEASE);
    return true;
}

int device_sm_count();    // of the current device (wkv56_chunked.cu)

// scalar (token-serial) v5/v6 kernels, wkv56_scalar.cu
size_t scalar_backward_workspace(const wkv_args_t *a);
// floor: decays floored at 0.005, as the chunked kernels do
int scalar_forward(const wkv_args_t *a, bool per_token_w, bool floor, cudaStream_t s);
int scalar_backward(const wkv_args_t *a, bool per_token_w, cudaStream_t s);

// chunked tensor-core v5/v6 kernels, wkv56_chunked.cu
bool chunked_supported(const wkv_args_t *a, bool per_token_w);
size_t chunked_forward_workspace(const wkv_args_t *a, bool per_token_w);
size_t chunked_backward_workspace(const wkv_args_t *a, bool per_token_w);

}  // namespace wkv
