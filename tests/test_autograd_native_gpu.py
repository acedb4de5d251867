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
