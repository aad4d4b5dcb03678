// Shared helpers of the PyTorch binding: error translation, the status words, small tensor helpers.
#pragma once
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include "wkv_internal.h"

namespace wkv_native {

using at::Tensor;
using OptTensor = c10::optional<Tensor>;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

constexpr int64_t HEAD = 64;

inline void check(int code, const char *what) {
    TORCH_CHECK(code == WKV_OK, what, ": ", wkv_error_string(code), " (code ", code, ")");
}
inline int dtype_code(at::ScalarType t) {
    switch (t) {
        case at::kFloat: return WKV_F32;
        case at::kBFloat16: return WKV_BF16;
        case at::kHalf: return WKV_F16;
        default: TORCH_CHECK_VALUE(false, "unsupported dtype ", t); return -1;
    }
}
inline void *ptr(const Tensor &t) { return t.defined() ? t.data_ptr() : nullptr; }
inline void *stream_of(const Tensor &t) { return at::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
inline Tensor contig(const Tensor &t) { return t.is_contiguous() ? t : t.contiguous(); }
inline Tensor as_contig(const Tensor &t, at::ScalarType dt) { return t.scalar_type() == dt ? contig(t) : t.to(dt).contiguous(); }
inline void require_cuda(std::initializer_list<const Tensor *> ts) {
    const Tensor *first = nullptr;
    for (const Tensor *t : ts) {
        if (!t->defined()) continue;
        TORCH_CHECK(t->is_cuda(), "wkv_b200 ops run on CUDA tensors only (there is no CPU path)");
        if (!first) first = t;
        TORCH_CHECK(t->device() == first->device(), "all tensors of one WKV call must live on the same device");
    }
}
inline Tensor bytes_like(const Tensor &t, size_t n) {
    return n ? at::empty({(int64_t)n}, t.options().dtype(at::kByte)) : Tensor();
}
// whether autograd will want a backward of a call on these tensors
inline bool wants_grad(std::initializer_list<const Tensor *> ts) {
    if (!at::GradMode::is_enabled()) return false;
    for (const Tensor *t : ts)
        if (t->defined() && t->requires_grad()) return true;
    return false;
}

// The device's status word: mapped host memory, written by a kernel only when one of its bounded waits
// runs out.  Looking at it costs one host load, so every call looks before it launches.
int *status_word(int device);
void poll_status(int device, bool wait);

}  // namespace wkv_native
