// The differentiable operators, as C++ autograd functions. For calls of a few tens of
// microseconds the host work of Python autograd functions (argument marshalling, autocast
// decorators, the interpreter lock in the backward thread) is most of the time: 112 us per forward +
// backward of 1000 queries against 40 us of kernels. Behaviour is that of the Python classes next
// to them in drivingsdk_b200/ops (which callers may still subclass, patch or apply):
//   * under autocast the attention operators run in float32 on cast inputs;
//   * an empty operand raises the reference's Exception;
//   * gradients are once-differentiable: using them in a graph raises;
//   * while torch.jit.trace records, the calls go through those classes, which the tracer sees (a
//     call that it does not see becomes a constant: the result for the example input).
// A call of the attention operators, the aggregation or max pooling whose gradient nobody asks for runs the
// forward without a node: building one takes 1.4 of the 9.2 us of a small inference call.
#include <ATen/FuncTorchTLS.h>
#include <ATen/autocast_mode.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/extension.h>

#include "bindings.h"

namespace sdk {
namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;

[[noreturn]] void raise_empty() {
    pybind11::gil_scoped_acquire gil;
    PyErr_SetString(PyExc_Exception, "Error! Input Tensor can not be a empty Tensor.\n");
    throw pybind11::error_already_set();
}

// custom_fwd(cast_inputs=torch.float32)
Tensor autocast_f32(const Tensor& t, bool on) {
    return on && t.is_floating_point() && t.is_cuda() && t.scalar_type() != at::kDouble
               ? t.to(at::kFloat)
               : t;
}

// @once_differentiable: where a graph of the gradients is asked for, they carry a node that
// raises when it is used.
variable_list once(variable_list grads, const Tensor& grad_out) {
    if (!at::GradMode::is_enabled() || !grad_out.requires_grad()) return grads;
    variable_list in;
    for (auto& g : grads) {
        Tensor t = g;
        if (t.defined()) {
            t = t.detach();
            t.requires_grad_(true);
        }
        in.push_back(t);
    }
    auto node = std::make_shared<torch::autograd::DelayedError>(
        "trying to differentiate twice a function that was marked with @once_differentiable",
        static_cast<int64_t>(in.size()));
    return (*node)(std::move(in));
}

// int32 or int64 level tables, both alike
void tables(Tensor& shapes, Tensor& starts) {
    const auto kind = shapes.scalar_type();
    if (kind == starts.scalar_type() && (kind == at::kInt || kind == at::kLong)) return;
    shapes = shapes.to(at::kInt);
    starts = starts.to(at::kInt);
}

// Whether a call can do without a node: no gradient and no tangent to carry, no functorch transform
// (which the node refuses). The forwards then get no context.
bool any_requires_grad(at::TensorList ts) {
    if (!at::GradMode::is_enabled()) return false;
    for (const Tensor& t : ts)
        if (t.defined() && t.requires_grad()) return true;
    return false;
}
bool without_node(at::TensorList ts) {
    if (any_requires_grad(ts) || at::functorch::functorchTLSAccessor() != nullptr) return false;
    for (const Tensor& t : ts)
        if (t.defined() && t._fw_grad(0).defined()) return false;
    return true;
}

struct Msda : Function<Msda> {
    static Tensor forward(AutogradContext* ctx, Tensor value, Tensor shapes, Tensor starts,
                          Tensor loc, Tensor attn) {
        const bool cast = at::autocast::is_autocast_enabled(at::kCUDA);
        value = autocast_f32(value, cast);
        if (value.numel() == 0 || shapes.numel() == 0 || attn.numel() == 0) raise_empty();
        tables(shapes, starts);
        loc = loc.to(value.scalar_type());
        attn = attn.to(value.scalar_type());
        Tensor out = msda_forward(value, shapes, starts, loc, attn);
        if (ctx) ctx->save_for_backward({value, shapes, starts, loc, attn});
        return out;
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        const auto s = ctx->get_saved_variables();
        auto [gv, gl, ga] = [&] {
            const at::NoGradGuard no_grad;
            return msda_backward(s[0], s[1], s[2], s[3], s[4], g[0]);
        }();
        return once({gv, Tensor(), Tensor(), gl, ga}, g[0]);
    }
};

struct Fused : Function<Fused> {
    static Tensor forward(AutogradContext* ctx, Tensor value, Tensor shapes, Tensor starts,
                          Tensor ref, Tensor off, Tensor logits) {
        const bool cast = at::autocast::is_autocast_enabled(at::kCUDA);
        value = autocast_f32(value, cast);
        if (value.numel() == 0 || shapes.numel() == 0 || logits.numel() == 0) raise_empty();
        tables(shapes, starts);
        ref = ref.to(value.scalar_type());
        off = off.to(value.scalar_type());
        logits = logits.to(value.scalar_type());
        Tensor out = msda_fused_forward(value, shapes, starts, ref, off, logits);
        if (ctx) ctx->save_for_backward({value, shapes, starts, ref, off, logits});
        return out;
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        const auto s = ctx->get_saved_variables();
        auto [gv, gr, go, gl] = [&] {
            const at::NoGradGuard no_grad;
            return msda_fused_backward(s[0], s[1], s[2], s[3], s[4], s[5], g[0]);
        }();
        return once({gv, Tensor(), Tensor(), gr, go, gl}, g[0]);
    }
};

struct Gka : Function<Gka> {
    static Tensor forward(AutogradContext* ctx, Tensor value, Tensor shapes, Tensor starts,
                          Tensor loc, Tensor attn) {
        TORCH_CHECK(value.dim() == 4, "geometric_kernel_attention: value [bs, keys, heads, dims] expected");
        // written in full by the kernel, with zeros if it refuses a level table
        Tensor out = at::empty({value.size(0), attn.size(1), value.size(2) * value.size(3)}, value.options());
        geometric_kernel_attention_forward(value, shapes, starts, loc, attn, out);
        if (ctx) ctx->save_for_backward({value, shapes, starts, loc, attn});
        return out;
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        const auto s = ctx->get_saved_variables();
        const at::NoGradGuard no_grad;
        auto [gv, ga] = geometric_kernel_attention_backward(s[0], s[1], s[2], s[3], s[4], g[0]);
        return {gv, Tensor(), Tensor(), Tensor(), ga};
    }
};

struct Aggregation : Function<Aggregation> {
    static Tensor forward(AutogradContext* ctx, Tensor feat, Tensor shape, Tensor start, Tensor loc,
                          Tensor wts) {
        if (feat.numel() == 0 || wts.numel() == 0) raise_empty();
        feat = feat.contiguous();
        shape = shape.contiguous().to(at::kInt);
        start = start.contiguous().to(at::kInt);
        loc = loc.contiguous();
        wts = wts.contiguous();
        Tensor out = deformable_aggregation(feat, shape, start, loc, wts);
        if (ctx) ctx->save_for_backward({feat, shape, start, loc, wts});
        return out;
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        const auto s = ctx->get_saved_variables();
        if (s[0].numel() == 0 || s[1].numel() == 0 || s[3].numel() == 0) raise_empty();
        const at::NoGradGuard no_grad;
        auto [gf, gl, gw] = deformable_aggregation_backward(s[0], s[1], s[2], s[3], s[4], g[0],
                                                            Tensor(), Tensor(), Tensor());
        return {gf, Tensor(), Tensor(), gl, gw};
    }
};

// the reference overwrites x only from this size up (mx_driving/ops/npu_add_relu.py:22)
constexpr int64_t kInPlaceMinNumel = 2000000;

struct AddRelu : Function<AddRelu> {
    static Tensor forward(AutogradContext* ctx, Tensor x, const Tensor& y, bool in_place) {
        Tensor out;
        if (in_place) {
            out = npu_add_relu(x, y);
            ctx->mark_dirty({x});
        } else {
            out = add_relu_out(x, y);
        }
        ctx->save_for_backward({out});
        return out;
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        const at::NoGradGuard no_grad;
        const Tensor r = npu_add_relu_grad(ctx->get_saved_variables()[0], g[0]);
        return {r, r, Tensor()};
    }
};

// Deformable convolution, modulated where `mask` is given (then `bias` may be). Keeps copies, so
// that the operands may be overwritten: the pair form its block and the weights, the fp32 form
// (other channel counts, mixed types) the channels-last tensors and the columns.
struct DeformConv : Function<DeformConv> {
    static Tensor forward(AutogradContext* ctx, Tensor x, Tensor offset, std::optional<Tensor> mask_opt,
                          Tensor weight, std::optional<Tensor> bias_opt, std::vector<int64_t> stride, std::vector<int64_t> padding,
                          std::vector<int64_t> dilation, int64_t groups, int64_t deformable_groups,
                          bool keep) {
        const Tensor mask = mask_opt.value_or(Tensor()), bias = bias_opt.value_or(Tensor());
        const bool modulated = mask.defined();
        const Conv conv{stride, padding, dilation, groups, deformable_groups};
        const auto kind = x.scalar_type();
        const bool alike = (kind == at::kFloat || kind == at::kHalf || kind == at::kBFloat16) &&
                           offset.scalar_type() == kind && weight.scalar_type() == kind &&
                           (!modulated || mask.scalar_type() == kind);
        ctx->saved_data["modulated"] = modulated;
        Tensor out, saved;
        std::vector<int64_t> shape;
        if (alike) std::tie(out, saved) = conv_forward(x, offset, mask, weight, bias, conv, keep, &shape);
        ctx->saved_data["shape"] = shape;   // empty: the fp32 form
        if (out.defined()) {
            if (keep) {
                ctx->save_for_backward({weight.clone(at::MemoryFormat::Contiguous), saved, bias});
            }
            return out;
        }
        const std::vector<int64_t> kernel{weight.size(2), weight.size(3)};
        auto nhwc = [](const Tensor& t) { return t.permute({0, 2, 3, 1}).contiguous(); };
        const Tensor nx = nhwc(x), noff = nhwc(offset), nw = nhwc(weight);
        const Tensor nmask = modulated ? nhwc(mask) : mask;
        Tensor columns;
        if (modulated) {
            std::tie(out, columns) = modulated_deformable_conv2d(
                nx, noff, nmask, nw, bias.defined() ? c10::optional<Tensor>(bias) : c10::nullopt, kernel, stride,
                padding, dilation, groups, deformable_groups, bias.defined() ? 1 : 0);
        } else {
            std::tie(out, columns) =
                deformable_conv2d(nx, noff, nw, kernel, stride, padding, dilation, groups, deformable_groups);
        }
        // (two entries each: checked by the call)
        ctx->saved_data["conv"] = std::vector<int64_t>{stride[0], stride[1], padding[0], padding[1], dilation[0],
                                                       dilation[1], groups, deformable_groups};
        ctx->save_for_backward({nw, columns, bias, nx, noff, nmask});
        return out;
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        const auto s = ctx->get_saved_variables();
        const auto shape = ctx->saved_data["shape"].toIntVector();
        const bool modulated = ctx->saved_data["modulated"].toBool(), with_bias = s[2].defined();
        ConvGrads r;
        {
            const at::NoGradGuard no_grad;
            if (!shape.empty()) {
                r = conv_backward(s[0], modulated, with_bias, s[1], g[0], shape);
                if (with_bias) r.bias = r.bias.to(s[2].scalar_type());
            } else {
                const auto c = ctx->saved_data["conv"].toIntVector();
                const std::vector<int64_t> kernel{s[0].size(1), s[0].size(2)}, stride{c[0], c[1]},
                    padding{c[2], c[3]}, dilation{c[4], c[5]};
                const Tensor go = g[0].permute({0, 2, 3, 1}).contiguous();
                if (modulated) {
                    std::tie(r.x, r.weight, r.bias, r.offset, r.mask) = modulated_deformable_conv2d_backward(
                        s[3], s[4], s[5], s[0], with_bias ? c10::optional<Tensor>(s[2]) : c10::nullopt, s[1], go,
                        kernel, stride, padding, dilation, c[6], c[7], with_bias ? 1 : 0);
                } else {
                    std::tie(r.x, r.weight, r.offset) = deformable_conv2d_backward(
                        s[3], s[0], s[4], s[1], go, kernel, stride, padding, dilation, c[6], c[7]);
                }
            }
        }
        return once({r.x, r.offset, r.mask, r.weight, r.bias, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()},
                    g[0]);
    }
};

// inference only, as in the reference: the result knows its input, but has no derivative
struct MaxPool : Function<MaxPool> {
    static Tensor forward(AutogradContext*, const Tensor& x, int64_t kernel, int64_t stride,
                          int64_t padding) {
        return npu_max_pool2d(x, static_cast<int>(kernel), static_cast<int>(stride),
                              static_cast<int>(padding));
    }
    static variable_list backward(AutogradContext*, variable_list) {
        TORCH_CHECK_NOT_IMPLEMENTED(false, "npu_max_pool2d has no backward");
    }
};

// `apply` of a Python class in drivingsdk_b200/ops.
template <typename... Args>
Tensor apply_class(const char* module, const char* name, const Args&... args) {
    pybind11::gil_scoped_acquire gil;
    const std::string path = std::string("drivingsdk_b200.ops.") + module;
    return pybind11::module_::import(path.c_str()).attr(name).attr("apply")(args...).template cast<Tensor>();
}
using torch::jit::tracer::isTracing;

Tensor msda(const Tensor& value, const Tensor& shapes, const Tensor& starts, const Tensor& loc,
            const Tensor& attn) {
    if (isTracing())
        return apply_class("multi_scale_deformable_attn", "MultiScaleDeformableAttnFunction", value, shapes,
                           starts, loc, attn);
    if (without_node({value, shapes, starts, loc, attn}))
        return Msda::forward(nullptr, value, shapes, starts, loc, attn);
    return Msda::apply(value, shapes, starts, loc, attn);
}
Tensor fused(const Tensor& value, const Tensor& shapes, const Tensor& starts, const Tensor& ref,
             const Tensor& off, const Tensor& logits) {
    if (isTracing())
        return apply_class("msda_fused", "MultiScaleDeformableAttnFusedFunction", value, shapes, starts, ref, off,
                           logits);
    if (without_node({value, shapes, starts, ref, off, logits}))
        return Fused::forward(nullptr, value, shapes, starts, ref, off, logits);
    return Fused::apply(value, shapes, starts, ref, off, logits);
}
Tensor gka(const Tensor& value, const Tensor& shapes, const Tensor& starts, const Tensor& loc,
           const Tensor& attn) {
    if (isTracing())
        return apply_class("geometric_kernel_attention", "GeometricKernelAttentionFunc", value, shapes, starts,
                           loc, attn);
    if (without_node({value, shapes, starts, loc, attn}))
        return Gka::forward(nullptr, value, shapes, starts, loc, attn);
    return Gka::apply(value, shapes, starts, loc, attn);
}
Tensor aggregation(const Tensor& feat, const Tensor& shape, const Tensor& start, const Tensor& loc,
                   const Tensor& wts) {
    if (isTracing())
        return apply_class("npu_deformable_aggregation", "AdsDeformableAggregation", feat, shape, start, loc, wts);
    if (without_node({feat, shape, start, loc, wts}))
        return Aggregation::forward(nullptr, feat, shape, start, loc, wts);
    return Aggregation::apply(feat, shape, start, loc, wts);
}
Tensor add_relu(const Tensor& x, const Tensor& y) {
    if (isTracing()) return apply_class("npu_add_relu", "AddReluFunction", x, y);
    const bool in_place = x.numel() >= kInPlaceMinNumel && x.is_contiguous() &&
                          !(x.is_leaf() && x.requires_grad());
    return AddRelu::apply(x, y, in_place);
}

using Pair = std::vector<int64_t>;
Tensor deform_conv(const Tensor& x, const Tensor& offset, const Tensor& weight, const Pair& stride,
                   const Pair& padding, const Pair& dilation, int64_t groups, int64_t deformable_groups) {
    if (isTracing())
        return apply_class("deform_conv2d", "DeformConv2dFunction", x, offset, weight, stride, padding, dilation,
                           groups, deformable_groups);
    return DeformConv::apply(x, offset, std::optional<Tensor>(), weight, std::optional<Tensor>(), stride, padding, dilation, groups,
                             deformable_groups, any_requires_grad({x, offset, weight}));
}
Tensor modulated_deform_conv(const Tensor& x, const Tensor& offset, const Tensor& mask, const Tensor& weight,
                             const c10::optional<Tensor>& bias, const Pair& stride, const Pair& padding,
                             const Pair& dilation, int64_t groups, int64_t deformable_groups) {
    if (isTracing())
        return apply_class("modulated_deform_conv2d", "ModulatedDeformConv2dFunction", x, offset, mask, weight, bias,
                           stride, padding, dilation, groups, deformable_groups);
    // custom_fwd(cast_inputs=torch.float32), the casts outside the function so that gradients
    // return through them
    const bool cast = at::autocast::is_autocast_enabled(at::kCUDA);
    const Tensor b = bias.has_value() ? *bias : Tensor();
    return DeformConv::apply(autocast_f32(x, cast), autocast_f32(offset, cast),
                             std::optional<Tensor>(autocast_f32(mask, cast)), autocast_f32(weight, cast),
                             b.defined() ? std::optional<Tensor>(autocast_f32(b, cast)) : std::nullopt, stride, padding,
                             dilation, groups, deformable_groups, any_requires_grad({x, offset, mask, weight, b}));
}
Tensor max_pool2d(const Tensor& x, int64_t kernel, int64_t stride, int64_t padding) {
    if (isTracing()) return apply_class("npu_max_pool2d", "MaxPool2d", x, kernel, stride, padding);
    if (without_node({x})) return MaxPool::forward(nullptr, x, kernel, stride, padding);
    return MaxPool::apply(x, kernel, stride, padding);
}

}  // namespace

void register_autograd(pybind11::module& m) {
    using release = pybind11::call_guard<pybind11::gil_scoped_release>;
    m.def("msda_autograd", &msda, release(), "differentiable multi_scale_deformable_attn");
    m.def("msda_fused_autograd", &fused, release(), "differentiable multi_scale_deformable_attn_fused");
    m.def("gka_autograd", &gka, release(), "differentiable geometric_kernel_attention");
    m.def("deformable_aggregation_autograd", &aggregation, release(), "differentiable deformable_aggregation");
    m.def("deform_conv2d_autograd", &deform_conv, release(), "differentiable deform_conv2d");
    m.def("modulated_deform_conv2d_autograd", &modulated_deform_conv, release(),
          "differentiable modulated_deform_conv2d");
    m.def("max_pool2d_autograd", &max_pool2d, release(), "npu_max_pool2d, known to autograd");
    m.def("add_relu_autograd", &add_relu, release(), "differentiable npu_add_relu");
}

}  // namespace sdk
