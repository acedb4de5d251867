"""Infinities reach what they contribute to and nothing else: corners outside the map take no part in
a gradient."""
import pytest
import torch

from drivingsdk_b200 import capi, workloads
from tests import parity

pytestmark = pytest.mark.gpu


def _same(name, got, want):
    assert torch.equal(torch.isnan(got), torch.isnan(want)), name
    assert torch.equal(torch.isinf(got), torch.isinf(want)), name
    fin = torch.isfinite(want)
    torch.testing.assert_close(got[fin], want[fin], rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D", [32, 24])
def test_sorted_backward_with_an_infinite_gradient(D, dtype):
    import drivingsdk_b200 as sdk
    w = workloads.Workload("inf", 1, 60, 2, D, ((3, 4), (1, 1)), 4, (-0.2, 1.2), seed=D)
    dev = parity.to_device(workloads.make_inputs(w, dtype), dtype)
    go = torch.ones(1, 60, 2 * D, dtype=dtype, device="cuda")
    go[0, ::3, 5] = float("inf")
    grads = []
    for sort in (0, 2):
        old = capi.load().msda_sm100_tune(capi.TUNE_SORT, sort)
        try:
            ts = [dev[k].detach().abs().requires_grad_() for k in ("value", "loc", "attn")]
            out = sdk.multi_scale_deformable_attn(ts[0], dev["shapes"], dev["starts"], *ts[1:])
            grads.append(torch.autograd.grad(out, ts, go))
        finally:
            capi.load().msda_sm100_tune(capi.TUNE_SORT, old)
    assert any(torch.isinf(g).any() for g in grads[0][1:])
    for name, want, got in zip(("value", "loc", "attn"), *grads):
        _same(name, got.float(), want.float())
