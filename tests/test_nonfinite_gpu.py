"""Infinities reach what they contribute to and nothing else: corners outside the map, and the lanes
of a row that is narrower than they are, take no part in a gradient."""
import pytest
import torch

from drivingsdk_b200 import capi, workloads
from tests import parity
from tests.test_da_gpu import _random_case

pytestmark = pytest.mark.gpu


def _same(name, got, want):
    assert torch.equal(torch.isnan(got), torch.isnan(want)), name
    assert torch.equal(torch.isinf(got), torch.isinf(want)), name
    fin = torch.isfinite(want)
    torch.testing.assert_close(got[fin], want[fin], rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D", [32, 24, 96, 256])
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


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D", [24, 32, 96, 256])
def test_sorted_fused_backward_with_values_that_are_not_finite(D, dtype):
    """Infinite gradients, reference points nowhere, masked logits (one task has no other), an infinite value."""
    import drivingsdk_b200 as sdk
    w = workloads.Workload("inf", 1, 60, 2, D, ((3, 4), (1, 1)), 4, (-0.2, 1.2), seed=D)
    dev = parity.to_device(workloads.make_inputs(w, dtype), dtype)
    g = torch.Generator(device="cuda").manual_seed(D)
    ref = torch.rand(1, 60, 2, 2, generator=g, device="cuda").to(dtype)
    ref[0, 7, 0, 0], ref[0, 8, 1, 1], ref[0, 9] = float("nan"), float("inf"), -float("inf")
    logits = torch.randn(1, 60, 2, 2, 4, generator=g, device="cuda").to(dtype)
    logits[0, ::5, :, 0, 1:] = -float("inf")
    logits[0, 11, 1] = -float("inf")
    value = dev["value"].abs() + 0.1
    value[0, 5, 1, D - 1] = float("inf")
    go = torch.ones(1, 60, 2 * D, dtype=dtype, device="cuda")
    go[0, ::3, 5] = float("inf")
    off = torch.randn(1, 60, 2, 2, 4, 2, generator=g, device="cuda").to(dtype)
    grads = []
    for sort in (0, 2):
        old = capi.load().msda_sm100_tune(capi.TUNE_SORT, sort)
        try:
            ts = [t.detach().requires_grad_() for t in (value, ref, off, logits)]
            out = sdk.multi_scale_deformable_attn_fused(ts[0], dev["shapes"], dev["starts"], *ts[1:])
            grads.append(torch.autograd.grad(out, ts, go))
        finally:
            capi.load().msda_sm100_tune(capi.TUNE_SORT, old)
    assert not torch.isfinite(grads[0][0]).all()
    for name, want, got in zip(("value", "ref", "off", "logits"), *grads):
        _same(name, got.float(), want.float())


def test_sorted_aggregation_with_an_infinite_gradient():
    c = _random_case(5, 1, 128, 9, 7, 4, [[(3, 4), (1, 2)]])
    c["feat"], c["grad_out"] = abs(c["feat"]) + 0.1, abs(c["grad_out"]) + 0.1
    c["wts"] = abs(c["wts"]) + 0.1
    c["grad_out"][0, ::2, 7] = float("inf")
    dev = {k: torch.from_numpy(c[k]).cuda() for k in c if k in ("feat", "shapes", "starts", "loc", "wts", "grad_out")}
    lib, stream = capi.load(), torch.cuda.current_stream().cuda_stream
    B, F, C = dev["feat"].shape
    dims = (B, F, C, *dev["wts"].shape[1:])
    ins = [dev[k].data_ptr() for k in ("feat", "shapes", "starts", "loc", "wts", "grad_out")]
    results = []
    for form in ("tasks", "sorted"):
        grads = [torch.empty_like(dev[k]) for k in ("feat", "loc", "wts")]
        outs = [g.data_ptr() for g in grads]
        if form == "tasks":
            capi.check(lib.da_sm100_backward(*ins, *outs, *dims, stream), form)
        else:
            ws = torch.empty(lib.da_sm100_backward_workspace_bytes(*dims), dtype=torch.uint8, device="cuda")
            capi.check(lib.da_sm100_backward_ws(*ins, *outs, ws.data_ptr(), ws.numel(), *dims, capi.F32, stream), form)
        results.append(grads)
    assert torch.isinf(results[0][1]).any()
    for name, want, got in zip(("feat", "loc", "wts"), *results):
        _same(name, got, want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("fused", [False, True])
def test_rows_that_leave_lanes_idle_with_an_infinite_value(dtype, fused):
    """An infinity in the last piece of a row: the row's own product with grad_out decides."""
    import drivingsdk_b200 as sdk
    D = 24
    w = workloads.Workload("inf", 1, 40, 2, D, ((3, 4), (2, 2)), 4, (0.2, 0.8), seed=3)
    dev = parity.to_device(workloads.make_inputs(w, dtype), dtype)
    value = dev["value"].abs() + 0.1
    value[0, 5, 0, D - 1] = float("inf")
    go = torch.ones(1, 40, 2 * D, dtype=dtype, device="cuda")
    call = sdk.multi_scale_deformable_attn
    rest = [dev["loc"], dev["attn"]]
    if fused:
        call = sdk.multi_scale_deformable_attn_fused
        rest = [torch.full((1, 40, 2, 2), 0.5, dtype=dtype, device="cuda"),
                ((dev["loc"].float() - 0.5) * 3).to(dtype), dev["attn"]]
    grads = []
    for odd in (True, False):   # at an odd address: channel by channel, no idle lanes
        v = value
        if odd:
            v = torch.empty(value.numel() + 1, dtype=dtype, device="cuda")[1:].view(value.shape).copy_(value)
        old = capi.load().msda_sm100_tune(capi.TUNE_SORT, 0)
        try:
            ts = [t.detach().requires_grad_() for t in (v, *rest)]
            out = call(ts[0], dev["shapes"], dev["starts"], *ts[1:])
            grads.append([g.float() for g in torch.autograd.grad(out, ts, go)])
        finally:
            capi.load().msda_sm100_tune(capi.TUNE_SORT, old)
    assert not torch.isfinite(grads[0][-1]).all()
    for i, (want, got) in enumerate(zip(*grads)):
        _same(i, got, want)
