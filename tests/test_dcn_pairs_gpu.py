"""The convolution's products over fp16 pairs, at the edges of their tiles and against the fp32 FMA
products: channel counts that fill 64, 128 and 256 wide tiles or leave remainders, groups whose row
blocks reach into the next group's, operands whose magnitudes differ by many orders between pixels (as
one norm over each result; pixel by pixel in test_dcn_range_gpu.py), channels-last gradients, Inf."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(x, off, mask, w, go, mode, stride=1, groups=1, dg=1, channels_last=False):
    import drivingsdk_b200 as sdk
    from drivingsdk_b200 import _C
    old = _C.dcn_use_tensor_cores(mode)
    try:
        ts = [t.clone().requires_grad_() for t in ((x, off, w) if mask is None else (x, off, mask, w))]
        if mask is None:
            out = sdk.deform_conv2d(*ts, stride, 1, 1, groups, dg)
        else:
            out = sdk.modulated_deform_conv2d(*ts, None, stride, 1, 1, groups, dg)
        g = go.contiguous(memory_format=torch.channels_last) if channels_last else go
        return (out.detach(), *torch.autograd.grad(out, ts, g))
    finally:
        _C.dcn_use_tensor_cores(old)


CASES = [
    # N, C, Co, H, W, stride, groups, dg, modulated
    (1, 8, 8, 3, 5, 1, 1, 1, True),
    (2, 24, 40, 9, 7, 1, 1, 1, False),
    (1, 64, 72, 17, 13, 2, 1, 4, True),
    (3, 96, 200, 11, 10, 1, 1, 1, True),
    (1, 128, 264, 12, 12, 1, 1, 2, True),
    (2, 64, 80, 10, 9, 1, 2, 1, True),
    (1, 512, 256, 13, 21, 1, 4, 1, False),
    # enough samples for the cell-sorted sampling: one and two passes of the lanes, slices, idle
    # lanes, several deformable groups
    (3, 104, 48, 62, 63, 1, 1, 1, True),
    (1, 264, 16, 111, 103, 1, 1, 1, True),
    (2, 320, 32, 41, 70, 1, 1, 2, False),
    (4, 256, 64, 55, 54, 1, 2, 2, True),
    # the sort's ways of keeping its counters that those do not take: split over a cluster (27226 cells),
    # one CTA per map
    (1, 104, 16, 164, 164, 1, 1, 1, True),
    (40, 104, 24, 20, 20, 1, 1, 1, True),
]


@pytest.mark.parametrize("case", CASES, ids=[f"c{c[1]}o{c[2]}g{c[6]}" for c in CASES])
def test_pairs_agree_with_fp32_products(case):
    N, C, Co, H, W, s, g, dg, modulated = case
    gen = torch.Generator(device="cuda").manual_seed(C + Co)
    r = lambda *shape: torch.randn(*shape, generator=gen, device="cuda")  # noqa: E731
    ho, wo = (H - 1) // s + 1, (W - 1) // s + 1
    # magnitudes spread over orders between images and pixels
    x = r(N, C, H, W) * torch.exp(3 * r(N, 1, H, W))
    off, mask = r(N, dg * 18, ho, wo), r(N, dg * 9, ho, wo).sigmoid() if modulated else None
    w, go = r(Co, C // g, 3, 3) / 30, r(N, Co, ho, wo) * torch.exp(3 * r(N, 1, ho, wo))
    for channels_last in (False, True):
        got = _run(x, off, mask, w, go, 1, s, g, dg, channels_last)
        want = _run(x, off, mask, w, go, 0, s, g, dg)
        for a, b in zip(got, want):
            assert a.shape == b.shape
            assert (a - b).norm() <= 1e-5 * b.norm() + 1e-30


def test_operands_may_be_overwritten_after_the_forward():
    import drivingsdk_b200 as sdk
    gen = torch.Generator(device="cuda").manual_seed(1)
    x, off, w = (torch.randn(*s, generator=gen, device="cuda") for s in
                 ((1, 16, 6, 6), (1, 18, 6, 6), (16, 16, 3, 3)))
    want = None
    for overwrite in (False, True):
        xs = x.clone().requires_grad_()
        inner, weight = xs * 1.0, w.clone().requires_grad_()
        out = sdk.deform_conv2d(inner, off, weight, 1, 1)
        if overwrite:
            inner.detach().zero_()
            weight.data.zero_()
        grads = torch.autograd.grad(out.sum(), (xs, weight))
        want = want or grads
        assert torch.equal(grads[1], want[1]) or (grads[1] - want[1]).norm() < 1e-6 * want[1].norm()
        assert (grads[0] - want[0]).norm() <= 1e-6 * want[0].norm()


def test_inf_stays_where_it_contributes():
    gen = torch.Generator(device="cuda").manual_seed(2)
    x = torch.randn(2, 16, 9, 9, generator=gen, device="cuda")
    off, w = torch.zeros(2, 18, 9, 9, device="cuda"), torch.randn(16, 16, 3, 3, generator=gen, device="cuda")
    go = torch.randn(2, 16, 9, 9, generator=gen, device="cuda")
    clean = _run(x, off, None, w, go, 1)[0]
    x[0, 3, 4, 4] = float("inf")
    out = _run(x, off, None, w, go, 1)[0]
    assert not torch.isfinite(out[0, :, 4, 4]).any()
    torch.testing.assert_close(out[1], clean[1], rtol=1e-5, atol=1e-5)
    torch.testing.assert_close(out[0, :, 0, :], clean[0, :, 0, :], rtol=1e-5, atol=1e-5)
