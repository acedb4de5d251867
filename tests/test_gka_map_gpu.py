"""Geometric kernel attention forward with the map in shared memory, against double-precision
gathers: every slice width it takes, ranges of a CTA that start and end inside maps, warps whose last
tasks are missing, one sample per task and the most, several levels, maps for two CTAs per SM and
for one, maps cut into slices, and one that is too large."""
import pytest
import torch

import drivingsdk_b200 as sdk
from tests import parity

pytestmark = pytest.mark.gpu

CASES = [
    # B, Q, H, D, levels, P
    (1, 4001, 1, 32, ((1, 1),), 1),
    (3, 1703, 5, 32, ((2, 3),), 3),
    (2, 2501, 4, 64, ((3, 5), (2, 2)), 15),
    (1, 1201, 3, 16, ((4, 4), (1, 7)), 32),
    (2, 9001, 4, 64, ((15, 25),), 15),
    (2, 5003, 8, 64, ((30, 26),), 9),     # fp32: 195 KB
    (1, 9001, 5, 64, ((30, 30),), 15),    # fp32: 225 KB, two slices
    (1, 9001, 5, 48, ((25, 25),), 15),    # fp32: 12 pieces, three slices; 16-bit: 6, another kernel
    (1, 21001, 2, 32, ((63, 57),), 15),   # fp32: slices of 224 KB, which leave no room for records
    (1, 7003, 5, 128, ((20, 20),), 15),   # fp32: 32 pieces; 16-bit: 16
]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("case", CASES, ids=[f"q{c[1]}d{c[3]}" for c in CASES])
def test_map_forward(case, dtype):
    B, Q, H, D, levels, P = case
    gen = torch.Generator().manual_seed(Q)
    shapes = torch.tensor(levels, dtype=torch.int32)
    sizes = shapes[:, 0] * shapes[:, 1]
    starts = (sizes.cumsum(0) - sizes).to(torch.int32)
    K, L = int(sizes.sum()), len(levels)
    value = torch.randn(B, K, H, D, generator=gen).to(dtype).cuda()
    attn = torch.rand(B, Q, H, L, P, generator=gen).to(dtype).cuda()
    extent = shapes.flip(-1).float()[:, None]   # (w, h); some samples fall outside
    loc = (torch.rand(B, Q, H, L, P, 2, generator=gen) * (extent + 4) - 2).floor().to(dtype).cuda()
    got = sdk.geometric_kernel_attention(value, shapes.cuda(), starts.cuda(), loc, attn)
    wh = shapes.flip(-1).long().cuda()[:, None]
    at = torch.minimum(loc.long().clamp(min=0), wh - 1)
    key = starts.long().cuda()[:, None] + at[..., 1] * wh[..., 0] + at[..., 0]
    want = torch.zeros(B, Q, H, D, dtype=torch.double, device="cuda")
    batch = torch.arange(B, device="cuda")[:, None, None]
    head = torch.arange(H, device="cuda")
    for i in range(L * P):
        k = key.flatten(3)[..., i]
        want += attn.flatten(3)[..., i, None].double() * value.double()[batch, k, head]
    if dtype != torch.float32:
        want = want.to(dtype).double()
    parity.assert_close("out", got, want.flatten(2).cpu().numpy(), parity.TOL[dtype])
