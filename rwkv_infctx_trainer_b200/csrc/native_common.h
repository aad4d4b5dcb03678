// Shared helpers of the PyTorch binding: error translation, the status words, small tensor helpers.
#pragma once
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
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
// a parameter as the kernels that read 16 bytes at a time take it (a copy when it starts elsewhere: parameters may be slices
// of one flat buffer)
inline Tensor as_param(const Tensor &t, at::ScalarType dt) {
    const Tensor c = as_contig(t, dt);
    return (reinterpret_cast<uintptr_t>(c.data_ptr()) & 15u) == 0 ? c : c.clone();
}
inline void require_cuda(std::initializer_list<const Tensor *> ts) {
    const Tensor *first = nullptr;
    for (const Tensor *t : ts) {
        if (!t->defined()) continue;
        TORCH_CHECK(t->is_cuda(), "wkv_b200 ops run on CUDA tensors only (there is no CPU path)");
        if (!first) first = t;
        TORCH_CHECK(t->device() == first->device(), "all tensors of one WKV call must live on the same device");
    }
}
// Fresh contiguous CUDA tensors, straight from the allocator: a call of the op makes six to ten, and through the
// dispatcher each costs half of a kernel launch.
inline Tensor fresh(at::IntArrayRef sizes, at::ScalarType dt, const Tensor &like) {
    return at::detail::empty_cuda(sizes, dt, like.device(), c10::nullopt);
}
inline Tensor fresh_like(const Tensor &t) { return fresh(t.sizes(), t.scalar_type(), t); }
inline Tensor bytes_like(const Tensor &t, size_t n) { return n ? fresh({(int64_t)n}, at::kByte, t) : Tensor(); }
// whether autograd will want a backward of a call on these tensors
inline bool wants_grad(std::initializer_list<const Tensor *> ts) {
    if (!at::GradMode::is_enabled()) return false;
    for (const Tensor *t : ts)
        if (t->defined() && t->requires_grad()) return true;
    return false;
}

// An autograd node with a list of saved tensors, written out (torch::autograd::Function builds maps and
// dictionaries around every call; at a few microseconds per kernel that shows).
struct OpNode : torch::autograd::Node {
    std::vector<torch::autograd::SavedVariable> saved;
    void keep(std::initializer_list<Tensor> ts) {
        saved.reserve(saved.size() + ts.size());
        for (const Tensor &t : ts) saved.emplace_back(t, false);
    }
    variable_list unpack() {
        std::lock_guard<std::mutex> hold(mutex_);
        variable_list r;
        r.reserve(saved.size());
        for (auto &v : saved) r.push_back(v.unpack());
        return r;
    }
    void release_variables() override {
        std::lock_guard<std::mutex> hold(mutex_);
        for (auto &v : saved) v.reset_data();
    }
};
template <class N>
std::shared_ptr<N> make_node(const variable_list &inputs) {
    std::shared_ptr<N> n(new N(), torch::autograd::deleteNode);
    n->set_next_edges(torch::autograd::collect_next_edges(inputs));
    return n;
}
// gradient in the type and shape its input has
inline Tensor as_input(Tensor g, at::ScalarType dt, at::IntArrayRef sizes) {
    if (!g.defined()) return g;
    if (g.scalar_type() != dt) g = g.to(dt);
    return g.sizes() == sizes ? g : g.view(sizes);
}

// The device's status word: mapped host memory, written by a kernel only when one of its bounded waits
// runs out.  Looking at it costs one host load, so every call looks before it launches.
int *status_word(int device);
void poll_status(int device, bool wait);

}  // namespace wkv_native
