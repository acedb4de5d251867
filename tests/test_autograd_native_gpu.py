"""The native autograd functions behave as the Python classes beside them."""
import pytest
import torch

from drivingsdk_b200 import workloads
from tests import parity

pytestmark = pytest.mark.gpu


def _leaves(dtype=torch.float32, queries=50):
    dev = parity.to_device(workloads.make_inputs(workloads.WORKLOADS["toy"].with_queries(queries), dtype), dtype)
    return dev["shapes"], dev["starts"], [dev[k].detach().requires_grad_() for k in ("value", "loc", "attn")]


@pytest.mark.parametrize("tables", [torch.int32, torch.int64, torch.int16])
@pytest.mark.parametrize("where", ["cuda", "cpu"])
def test_native_and_class_agree(tables, where):
    import drivingsdk_b200 as sdk
    shapes, starts, (v, l, a) = _leaves()
    shapes, starts = shapes.to(where, tables), starts.to(where, tables)
    for fn in (sdk.multi_scale_deformable_attn, sdk.MultiScaleDeformableAttnFunction.apply):
        out = fn(v, shapes, starts, l, a)
        grads = torch.autograd.grad(out, (v, l, a), torch.ones_like(out))
        if fn is sdk.multi_scale_deformable_attn:
            want, want_grads = out, grads
    assert torch.equal(out, want)
    torch.testing.assert_close(grads[0], want_grads[0], rtol=1e-5, atol=1e-5)
    assert torch.equal(grads[1], want_grads[1]) and torch.equal(grads[2], want_grads[2])


def test_gradients_are_once_differentiable():
    import drivingsdk_b200 as sdk
    shapes, starts, (v, l, a) = _leaves()
    out = sdk.multi_scale_deformable_attn(v, shapes, starts, l, a)
    go = torch.ones_like(out, requires_grad=True)
    (gv,) = torch.autograd.grad(out, v, go, create_graph=True)
    with pytest.raises(RuntimeError, match="once_differentiable"):
        gv.sum().backward()


def test_autocast_runs_in_float32_and_gradients_keep_the_input_type():
    import drivingsdk_b200 as sdk
    shapes, starts, (v, l, a) = _leaves(torch.float16)
    with torch.autocast("cuda", dtype=torch.float16):
        out = sdk.multi_scale_deformable_attn(v, shapes, starts, l, a)
    assert out.dtype == torch.float32
    assert all(g.dtype == torch.float16 for g in torch.autograd.grad(out.sum(), (v, l, a)))


def test_empty_operand_raises_the_references_exception():
    import drivingsdk_b200 as sdk
    shapes, starts, (v, l, a) = _leaves()
    with pytest.raises(Exception, match="empty Tensor") as e:
        sdk.multi_scale_deformable_attn(v[:, :0], shapes, starts, l, a)
    assert type(e.value) is Exception


def test_add_relu_in_place_under_autograd():
    import drivingsdk_b200 as sdk
    base = torch.randn(2, 1000, 1001, device="cuda", requires_grad=True)
    y = torch.randn_like(base).requires_grad_()
    x = base * 1.0
    out = sdk.npu_add_relu(x, y)
    assert out.data_ptr() == x.data_ptr()
    gx, gy = torch.autograd.grad(out.sum(), (base, y))
    assert torch.equal(gx, (out > 0).float()) and torch.equal(gx, gy)


def test_convolution_wants_two_strides():
    import drivingsdk_b200 as sdk
    for channels in (8, 6):   # the native form, and the fp32 form
        x, off, w = (torch.randn(*n, device="cuda") for n in ((1, channels, 5, 5), (1, 18, 5, 5), (8, channels, 3, 3)))
        for stride in ((1,), (1, 1, 1)):
            with pytest.raises(RuntimeError, match="two entries"):
                sdk.deform_conv2d(x, off, w, stride, 1)


def _traced_calls():
    import drivingsdk_b200 as sdk
    shapes, starts, (v, l, a) = _leaves()
    r = lambda *s: torch.randn(*s, device="cuda")  # noqa: E731
    yield "msda", lambda v, l, a: sdk.multi_scale_deformable_attn(v, shapes, starts, l, a), (v, l, a)
    off, ref = r(*l.shape), torch.rand(l.shape[0], l.shape[1], l.shape[3], 2, device="cuda")
    yield "fused", lambda v, f, o, a: sdk.multi_scale_deformable_attn_fused(v, shapes, starts, f, o, a), \
        (v, ref, off, a)
    tables = torch.tensor([[4, 5]], device="cuda"), torch.tensor([0], device="cuda")
    loc = torch.randint(0, 4, (1, 6, 2, 1, 3, 2), device="cuda").float()
    yield "gka", lambda v, a: sdk.geometric_kernel_attention(v, *tables, loc, a), (r(1, 20, 2, 8), r(1, 6, 2, 1, 3))
    maps = torch.tensor([[[4, 5]]], device="cuda"), torch.tensor([[0]], device="cuda")
    yield "da", lambda f, l, w: sdk.deformable_aggregation(f, *maps, l, w), \
        (r(1, 20, 32), torch.rand(1, 3, 2, 1, 2, device="cuda"), r(1, 3, 2, 1, 1, 8))
    conv = r(1, 8, 5, 5), r(1, 18, 5, 5), r(8, 8, 3, 3)
    yield "dcn", lambda x, o, w: sdk.deform_conv2d(x, o, w, 1, 1), conv
    yield "mdcn", lambda x, o, m, w, b: sdk.modulated_deform_conv2d(x, o, m, w, b, 1, 1), \
        (conv[0], conv[1], r(1, 9, 5, 5), conv[2], r(8))
    yield "add_relu", sdk.npu_add_relu, (r(3, 7), r(3, 7))
    yield "max_pool", lambda x: sdk.npu_max_pool2d(x, 3, 2, 1), (r(1, 2, 9, 9),)


def test_traced_operators_follow_their_inputs():
    """torch.jit.trace: the operators are in the graph, and not their results for the example."""
    for name, fn, args in _traced_calls():
        args = tuple(t.detach() for t in args)
        traced = torch.jit.trace(fn, args, check_trace=False)
        others = tuple(t.roll(1, 0) * 0.9 for t in args)
        torch.testing.assert_close(traced(*others), fn(*others), msg=lambda m, n=name: f"{n}: {m}")
