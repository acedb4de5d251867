"""Attention backwards where memory has no room for the workspace of their sorted form: they run in the form
that needs none, as they did before there was another, and give the same gradients."""
import pytest
import torch

from drivingsdk_b200 import _C, capi
from tests import parity

pytestmark = pytest.mark.gpu

B, Q, H, D, P, LEVELS = 1, 240000, 8, 32, 4, ((30, 40), (15, 20), (8, 10), (4, 5))   # 30.7 M samples


def _calls(op, dtype):
    g = torch.Generator(device="cuda").manual_seed(3)
    L, K = len(LEVELS), sum(h * w for h, w in LEVELS)
    shapes = torch.tensor(LEVELS, dtype=torch.int32)
    starts = torch.cat([torch.zeros(1, dtype=torch.int32), shapes.prod(1).cumsum(0)[:-1].int()]).cuda()
    shapes = shapes.cuda()
    torch.cuda.empty_cache()   # (no input in a larger block, whose rest would be room)
    kind = dict(generator=g, device="cuda", dtype=dtype)
    value, go = torch.rand(B, K, H, D, **kind), torch.randn(B, Q, H * D, **kind)
    logits, ref, off = (torch.rand(*s, **kind) for s in ((B, Q, H, L, P), (B, Q, L, 2), (B, Q, H, L, P, 2)))
    if op == "gka":
        off.mul_(40).floor_()
    dims = (B, K, H, D, L, Q, P, capi.dtype_code(dtype))
    lib = capi.load()
    return {"msda": (lambda: _C.multi_scale_deformable_attn_backward(value, shapes, starts, off, logits, go),
                     lib.msda_sm100_backward_sorted_workspace_bytes(*dims)),
            "fused": (lambda: _C.msda_fused_backward(value, shapes, starts, ref, off, logits, go),
                      lib.msda_sm100_fused_backward_sorted_workspace_bytes(*dims)),
            "gka": (lambda: _C.geometric_kernel_attention_backward(value, shapes, starts, off, logits, go),
                    lib.gka_sm100_backward_sorted_workspace_bytes(*dims))}


def _count(call):
    before = capi.load().msda_sm100_launch_count()
    got = call()
    torch.cuda.synchronize()
    return got, capi.load().msda_sm100_launch_count() - before


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("op", ["msda", "fused", "gka"])
def test_no_room_for_the_sorted_form(op, dtype):
    call, workspace = _calls(op, dtype)[op]
    want, launches = _count(call)
    convert = 0 if dtype == torch.float32 else 1
    assert launches == (4 if op == "fused" else 2) + convert
    results = sum(t.numel() * t.element_size() for t in want if t is not None)
    want = [t.cpu() for t in want]
    torch.cuda.empty_cache()
    room = torch.cuda.memory_reserved() + results + workspace // 2 + (24 << 20)
    assert workspace // 2 > 48 << 20
    torch.cuda.set_per_process_memory_fraction(room / torch.cuda.get_device_properties(0).total_memory)
    try:
        got, launches = _count(call)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert launches == 1 + convert
    # sums of n <= 1 M signed products in another order: off by some n * 2^-24 against a largest of some
    # 4 * sqrt(n), so 1.5e-5; 16-bit results may round to a neighbour
    tol = 1e-4 if dtype == torch.float32 else parity.TOL[dtype]
    for a, b in zip(got, want):
        assert (a.cpu().float() - b.float()).abs().max() <= tol * b.float().abs().max()
