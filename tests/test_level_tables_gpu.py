"""Level tables that the operators refuse: on the host before anything is launched, or in the kernel
where the host cannot read them."""
import pytest
import torch

from drivingsdk_b200 import capi

pytestmark = pytest.mark.gpu


def _tables(kind):
    cuda32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    shapes, starts = cuda32([[2, 3], [1, 2]]), cuda32([0, 6])
    return {"starts on the host": (shapes, starts.cpu()), "shapes on the host": (shapes.cpu(), starts),
            "int32 and int64": (shapes, starts.long()), "int64 and int32": (shapes.long(), starts),
            "int16": (shapes.short(), starts.short())}[kind]


@pytest.mark.parametrize("kind", ["starts on the host", "shapes on the host"])
def test_kernel_attention_wants_its_tables_together(kind):
    import drivingsdk_b200 as sdk
    from drivingsdk_b200 import _C
    value, attn = torch.zeros(1, 8, 1, 8, device="cuda"), torch.zeros(1, 3, 1, 2, 2, device="cuda")
    loc, go = torch.zeros(1, 3, 1, 2, 2, 2, device="cuda"), torch.zeros(1, 3, 8, device="cuda")
    with pytest.raises(RuntimeError, match="same device"):
        sdk.geometric_kernel_attention(value, *_tables(kind), loc, attn)
    with pytest.raises(RuntimeError, match="same device"):
        _C.geometric_kernel_attention_backward(value, *_tables(kind), loc, attn, go)


@pytest.mark.parametrize("kind", ["int32 and int64", "int64 and int32", "int16"])
def test_exported_functions_take_int32_tables(kind):
    from drivingsdk_b200 import _C
    value, logits = torch.zeros(1, 8, 1, 8, device="cuda"), torch.zeros(1, 3, 1, 2, 2, device="cuda")
    loc, ref = torch.zeros(1, 3, 1, 2, 2, 2, device="cuda"), torch.zeros(1, 3, 2, 2, device="cuda")
    go = torch.zeros(1, 3, 8, device="cuda")
    for call in (lambda s, t: _C.msda_fused_forward(value, s, t, ref, loc, logits),
                 lambda s, t: _C.msda_fused_backward(value, s, t, ref, loc, logits, go),
                 lambda s, t: _C.multi_scale_deformable_attn(value, s, t, loc, logits),
                 lambda s, t: _C.multi_scale_deformable_attn_backward(value, s, t, loc, logits, go)):
        for place in ("cuda", "cpu"):
            with pytest.raises(RuntimeError, match="int32 tensor expected"):
                call(*(t.to(place) for t in _tables(kind)))


@pytest.mark.parametrize("Q", [5, 4000], ids=["gather", "map"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_refused_table_leaves_zeros(Q, dtype):
    """geometric_kernel_attention's output is zero where the kernel refuses the table (its memory
    is not what an earlier tensor left there)."""
    import drivingsdk_b200 as sdk
    value = torch.ones(2, 12, 4, 64, device="cuda", dtype=dtype)
    attn = torch.ones(2, Q, 4, 1, 15, device="cuda", dtype=dtype)
    loc = torch.zeros(2, Q, 4, 1, 15, 2, device="cuda", dtype=dtype)
    shapes = torch.tensor([[100, 100]], device="cuda")   # more pixels than there are keys
    starts = torch.zeros(1, dtype=torch.int64, device="cuda")
    assert capi.load().msda_sm100_device_status(1) == 0
    stale = torch.full((2, Q, 256), 7.0, device="cuda", dtype=dtype)
    del stale
    out = sdk.geometric_kernel_attention(value, shapes, starts, loc, attn)
    assert capi.load().msda_sm100_device_status(1) == 4
    assert not out.any()
