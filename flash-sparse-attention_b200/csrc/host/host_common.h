// Shared by the native host code: tensors in, C-ABI calls out (include/fsa_sm100.h).  Everything here runs on the calling
// thread and never synchronises.
#pragma once
#include <torch/extension.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include "../../../include/fsa_sm100.h"

namespace fsa_host {

using at::Tensor;

inline void check(int rc, const char* what) {
    if (rc == FSA_OK) return;
    if (rc == FSA_ERR_BAD_ARG || rc == FSA_ERR_UNSUPPORTED) TORCH_CHECK_VALUE(false, what, ": ", fsa_error_string(rc));
    if (rc == FSA_ERR_CUDA)
        TORCH_CHECK(false, what, ": ", fsa_error_string(rc), " (cudaError ", fsa_last_cuda_error(), " at fsa_api.cu:", fsa_last_cuda_error_line(), ")");
    TORCH_CHECK(false, what, ": ", fsa_error_string(rc));
}

inline int dtype_code(const Tensor& t) {
    TORCH_CHECK_TYPE(t.scalar_type() == at::kBFloat16 || t.scalar_type() == at::kHalf, "bf16 or fp16 expected, got ", t.scalar_type());
    return t.scalar_type() == at::kBFloat16 ? FSA_DTYPE_BF16 : FSA_DTYPE_FP16;
}

inline void* stream_of(const Tensor& t) { return (void*)c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

// Can the kernels read this [N, H, D] tensor in place?  (packed: the heads of a token are adjacent, which the K/V maps need)
inline bool rows_ok(const Tensor& t, bool packed) {
    return t.stride(2) == 1 && ((uintptr_t)t.data_ptr() & 15) == 0 && t.stride(0) % 8 == 0 && t.stride(1) % 8 == 0 &&
           (!packed || t.stride(1) == t.size(2));
}
inline Tensor rows(const Tensor& t, bool packed = false) { return rows_ok(t, packed) ? t : t.contiguous(); }

// Memory straight from the allocator: a layer's step makes some fifty tensors, and the dispatcher's share of each is as long as the rest.
inline Tensor fresh(at::IntArrayRef shape, at::ScalarType type, const Tensor& like) {
    return Tensor(at::detail::empty_cuda(shape, type, like.device(), std::nullopt));
}
inline Tensor fresh(at::IntArrayRef shape, const Tensor& like) { return fresh(shape, like.scalar_type(), like); }
inline Tensor fresh_like(const Tensor& like) { return fresh(like.sizes(), like); }      // (contiguous)
inline Tensor bytes(int64_t n, const Tensor& like) { return fresh({std::max<int64_t>(n, 16)}, at::kByte, like); }
inline Tensor f32(at::IntArrayRef shape, const Tensor& like) { return fresh(shape, at::kFloat, like); }
inline Tensor i32(at::IntArrayRef shape, const Tensor& like) { return fresh(shape, at::kInt, like); }
inline const int32_t* iptr(const Tensor& t) { return t.defined() ? t.data_ptr<int32_t>() : nullptr; }
inline void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

inline bool wants_grad(std::initializer_list<const Tensor*> ts) {
    if (!at::GradMode::is_enabled()) return false;
    for (auto* t : ts)
        if (t->defined() && t->requires_grad()) return true;
    return false;
}

// selected attention (sel_host.cpp): o, lse and the index; dq, dk, dv from delta = sum_d o dO
std::tuple<Tensor, Tensor, Tensor> sel_fwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& idx, int64_t bs, const Tensor& cu,
                                           double scale);
std::tuple<Tensor, Tensor, Tensor> sel_bwd_delta(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& lse, const Tensor& dout,
                                                 const float* delta, const Tensor& idx, int64_t bs, const Tensor& cu, double scale,
                                                 const Tensor& ws);

// FSA_CHECK_STATUS=1: after their launches the operators read the status words of their kernels (one synchronisation each) and
// raise when a bounded wait ran out.
bool checking_status();
void check_status(const void* word, const Tensor& like, const char* what);

void bind_sel(pybind11::module& m);
void bind_decode(pybind11::module& m);
void bind_layer(pybind11::module& m);

}  // namespace fsa_host
