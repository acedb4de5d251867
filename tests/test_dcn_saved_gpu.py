"""The convolution's saved block, and the limits of its native form."""
import ctypes

import pytest
import torch

from drivingsdk_b200 import capi

pytestmark = pytest.mark.gpu


class Shape(ctypes.Structure):
    _fields_ = [(n, ctypes.c_int) for n in ("N", "H", "W", "C", "Ho", "Wo", "Co", "kh", "kw", "stride_h", "stride_w",
                                            "pad_h", "pad_w", "dil_h", "dil_w", "groups", "deform_groups")]


def test_backward_only_reads_what_the_forward_saved():
    N, C, H, W = 8, 104, 62, 63    # samples enough for the cell-sorted sampling, on more warps than fit
    s = Shape(N, H, W, C, H, W, 16, 3, 3, 1, 1, 1, 1, 1, 1, 1, 1)
    lib, stream, ref = capi.load(), torch.cuda.current_stream().cuda_stream, ctypes.byref(s)
    r = lambda *shape: torch.randn(*shape, device="cuda")  # noqa: E731
    x, off, mask, w, go = r(N, C, H, W), r(N, 18, H, W), r(N, 9, H, W), r(16, C, 3, 3), r(N, 16, H, W)
    block = lambda n: torch.zeros(n, dtype=torch.uint8, device="cuda")  # noqa: E731
    saved, out = block(lib.dcn_sm100_saved_bytes(ref, 0, 1)), r(N, H, W, 16)
    ws = block(lib.dcn_sm100_nchw_workspace_bytes(ref, 0, 1, 0))
    ptr = lambda *ts: [t.data_ptr() for t in ts]  # noqa: E731
    capi.check(lib.dcn_sm100_forward_nchw(x.data_ptr(), 0, *ptr(off, mask, w), None, *ptr(out, saved), saved.numel(),
                                          ws.data_ptr(), ws.numel(), ref, 0, 1, stream), "forward")
    before = saved.clone()
    ws = block(lib.dcn_sm100_nchw_workspace_bytes(ref, 0, 1, 1))
    gx, goff, gmask, gw = r(N, H, W, C), r(N, H, W, 18), r(N, H, W, 9), r(16, 3, 3, C)
    capi.check(lib.dcn_sm100_backward_nchw(w.data_ptr(), go.data_ptr(), 0, *ptr(saved, gx, goff, gmask, gw), None,
                                           ws.data_ptr(), ws.numel(), ref, 0, stream), "backward")
    assert torch.equal(saved, before)


def test_more_images_than_a_grid_has_planes():
    import drivingsdk_b200 as sdk
    N = 65537
    torch.manual_seed(5)
    x, off = torch.randn(N, 8, 2, 2, device="cuda"), torch.randn(N, 18, 2, 2, device="cuda")
    w = torch.randn(8, 8, 3, 3, device="cuda")
    ts = [t.requires_grad_() for t in (x, off, w)]
    out = sdk.deform_conv2d(*ts, 1, 1)
    go = torch.randn_like(out)
    got = torch.autograd.grad(out, ts, go)
    parts = []
    for half in (slice(0, 30000), slice(30000, N)):
        p = [x.detach()[half].requires_grad_(), off.detach()[half].requires_grad_(), w.detach().requires_grad_()]
        o = sdk.deform_conv2d(*p, 1, 1)
        parts.append((o.detach(), *torch.autograd.grad(o, p, go[half])))
    want = [torch.cat([a[i] for a in parts]) for i in range(3)] + [parts[0][3] + parts[1][3]]
    for name, a, b in zip(("out", "grad_x", "grad_offset", "grad_weight"), (out, *got), want):
        # grad_weight may be one serial fp32 sum over n = 262148 pixels, whose rounding is off by some
        # 2^-24 * sqrt(n / 6) = 1.2e-5 of the result; four times that
        assert (a - b).norm() <= (5e-5 if name == "grad_weight" else 1e-5) * b.norm(), name
