// The operator calls of binding.cpp that the autograd functions (autograd.cpp) use. Level tables
// may be int32 or int64.
#pragma once

#include <ATen/ATen.h>

#include <tuple>

namespace sdk {
at::Tensor msda_forward(const at::Tensor& value, const at::Tensor& shapes, const at::Tensor& starts,
                        const at::Tensor& loc, const at::Tensor& attn);
std::tuple<at::Tensor, at::Tensor, at::Tensor> msda_backward(
    const at::Tensor& value, const at::Tensor& shapes, const at::Tensor& starts,
    const at::Tensor& loc, const at::Tensor& attn, const at::Tensor& grad_out);
at::Tensor add_relu_out(const at::Tensor& x, const at::Tensor& y);
}  // namespace sdk

at::Tensor msda_fused_forward(const at::Tensor& value, const at::Tensor& shapes,
                              const at::Tensor& starts, const at::Tensor& ref,
                              const at::Tensor& off, const at::Tensor& logits);
std::tuple<at::Tensor, at::Tensor, at::Tensor, at::Tensor> msda_fused_backward(
    const at::Tensor& value, const at::Tensor& shapes, const at::Tensor& starts,
    const at::Tensor& ref, const at::Tensor& off, const at::Tensor& logits,
    const at::Tensor& grad_out);
void geometric_kernel_attention_forward(const at::Tensor& value, const at::Tensor& shapes,
                                        const at::Tensor& starts, const at::Tensor& loc,
                                        const at::Tensor& attn, at::Tensor& output);
std::tuple<at::Tensor, at::Tensor> geometric_kernel_attention_backward(
    const at::Tensor& value, const at::Tensor& shapes, const at::Tensor& starts,
    const at::Tensor& loc, const at::Tensor& attn, const at::Tensor& grad_out);
at::Tensor deformable_aggregation(const at::Tensor& feat, const at::Tensor& shape,
                                  const at::Tensor& start, const at::Tensor& loc,
                                  const at::Tensor& wts);
std::tuple<at::Tensor, at::Tensor, at::Tensor> deformable_aggregation_backward(
    const at::Tensor& feat, const at::Tensor& shape, const at::Tensor& start,
    const at::Tensor& loc, const at::Tensor& wts, const at::Tensor& grad_out,
    const at::Tensor& grad_feat, const at::Tensor& grad_loc, const at::Tensor& grad_wts);
at::Tensor npu_add_relu(at::Tensor& x, const at::Tensor& y);
at::Tensor npu_add_relu_grad(const at::Tensor& self, const at::Tensor& grad_output);
at::Tensor npu_max_pool2d(const at::Tensor& x, int kernel_size, int stride, int padding);
