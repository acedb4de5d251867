// The operator calls of binding.cpp that the autograd functions (autograd.cpp) use. Level tables
// may be int32 or int64.
#pragma once

#include <ATen/ATen.h>

#include <tuple>
#include <vector>

namespace sdk {
at::Tensor msda_forward(const at::Tensor& value, const at::Tensor& shapes, const at::Tensor& starts,
                        const at::Tensor& loc, const at::Tensor& attn);
std::tuple<at::Tensor, at::Tensor, at::Tensor> msda_backward(
    const at::Tensor& value, const at::Tensor& shapes, const at::Tensor& starts,
    const at::Tensor& loc, const at::Tensor& attn, const at::Tensor& grad_out);
// Deformable convolution over fp16 pairs, from NCHW tensors of one type. conv_forward returns the
// output and the block that conv_backward needs, or undefined tensors where the form does not
// apply; `keep`: a backward may follow; `shape` receives the sizes for conv_backward. Nothing of x, offset and mask is needed
// later, so callers may overwrite them.
struct Conv {
    std::vector<int64_t> stride, padding, dilation;
    int64_t groups, deformable_groups;
};
struct ConvGrads {
    at::Tensor x, offset, mask, weight, bias;   // fp32 values in `weight`'s type; bias fp32
};
std::tuple<at::Tensor, at::Tensor> conv_forward(const at::Tensor& x, const at::Tensor& offset,
                                                const at::Tensor& mask, const at::Tensor& weight,
                                                const at::Tensor& bias, const Conv& conv, bool keep,
                                                std::vector<int64_t>* shape);
ConvGrads conv_backward(const at::Tensor& weight, bool modulated, bool with_bias, const at::Tensor& saved,
                        const at::Tensor& grad_out, const std::vector<int64_t>& shape);
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
std::tuple<at::Tensor, at::Tensor> deformable_conv2d(
    const at::Tensor& input, const at::Tensor& offset, const at::Tensor& weight,
    at::IntArrayRef kernel_size, at::IntArrayRef stride, at::IntArrayRef padding,
    at::IntArrayRef dilation, int64_t groups, int64_t deformable_groups);
std::tuple<at::Tensor, at::Tensor, at::Tensor> deformable_conv2d_backward(
    const at::Tensor& input, const at::Tensor& weight, const at::Tensor& offset,
    const at::Tensor& offset_output, const at::Tensor& grad_y, at::IntArrayRef kernel_size,
    at::IntArrayRef stride, at::IntArrayRef padding, at::IntArrayRef dilation, int64_t groups,
    int64_t deformable_groups);
std::tuple<at::Tensor, at::Tensor> modulated_deformable_conv2d(
    const at::Tensor& input, const at::Tensor& offset, const at::Tensor& mask,
    const at::Tensor& weight, const c10::optional<at::Tensor>& bias_opt,
    at::IntArrayRef kernel_size, at::IntArrayRef stride, at::IntArrayRef padding,
    at::IntArrayRef dilation, int64_t groups, int64_t deformable_groups, int64_t with_bias);
std::tuple<at::Tensor, at::Tensor, at::Tensor, at::Tensor, at::Tensor>
modulated_deformable_conv2d_backward(
    const at::Tensor& input, const at::Tensor& offset, const at::Tensor& mask,
    const at::Tensor& weight, const c10::optional<at::Tensor>& bias_opt,
    const at::Tensor& offset_output, const at::Tensor& grad_y, at::IntArrayRef kernel_size,
    at::IntArrayRef stride, at::IntArrayRef padding, at::IntArrayRef dilation, int64_t groups,
    int64_t deformable_groups, int64_t with_bias);
