"""Deformable aggregation backward over cell-sorted samples and the typed forward, at the edges of
their tiles: rows of one and two passes of the lanes, idle lanes, one-pixel maps, points outside."""
import pytest
import torch

from drivingsdk_b200 import capi
from oracle import msda_oracle
from tests import parity
from tests.test_da_gpu import _random_case

pytestmark = pytest.mark.gpu

CASES = [  # B, C, A, Pts, G, maps
    (1, 68, 3, 5, 17, [[(1, 1), (2, 3)]]),
    (2, 96, 7, 9, 6, [[(5, 4)], [(3, 6)]]),
    (1, 128, 40, 33, 4, [[(4, 4), (2, 2)]]),
    (2, 192, 5, 7, 6, [[(9, 3), (1, 5)], [(2, 2), (7, 7)]]),
    (1, 256, 60, 13, 8, [[(6, 9), (3, 5), (2, 3), (1, 2)]] * 3),
]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("case", CASES, ids=[f"c{c[1]}" for c in CASES])
def test_sorted_backward(case, dtype):
    B, C, A, Pts, G, maps = case
    c = _random_case(C, B, C, A, Pts, G, maps)
    for k in ("feat", "loc", "wts", "grad_out"):
        c[k] = torch.from_numpy(c[k]).to(dtype).float().numpy()
    lib = capi.load()
    dev = {k: torch.from_numpy(c[k]).cuda().to(dtype) for k in ("feat", "loc", "wts", "grad_out")}
    shapes, starts = torch.from_numpy(c["shapes"]).cuda(), torch.from_numpy(c["starts"]).cuda()
    dims = (B, c["feat"].shape[1], C, A, Pts, len(maps), len(maps[0]), G)
    gf, gl, gw = (torch.empty(c[k].shape, device="cuda") for k in ("feat", "loc", "wts"))
    nbytes = lib.da_sm100_backward_workspace_bytes(*dims)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    ptrs = [dev["feat"], shapes, starts, dev["loc"], dev["wts"], dev["grad_out"], gf, gl, gw, ws]
    capi.check(lib.da_sm100_backward_ws(*(t.data_ptr() for t in ptrs), nbytes, *dims,
                                        capi.dtype_code(dtype), stream), "da backward")
    wf, wl, ww = msda_oracle.da_backward(c["feat"], c["shapes"], c["starts"], c["loc"], c["wts"],
                                         c["grad_out"])
    parity.assert_close("grad_feat", gf, wf, 1e-4)
    parity.assert_close("grad_weights", gw, ww, 1e-4)
    parity.assert_close("grad_loc", gl, wl, 1e-3)
    if C in (128, 256):
        out = torch.empty(B, A, C, device="cuda")
        capi.check(lib.da_sm100_forward_typed(
            *(t.data_ptr() for t in ptrs[:5]), out.data_ptr(), *dims, capi.dtype_code(dtype), stream), "fwd")
        want = msda_oracle.da_forward(c["feat"], c["shapes"], c["starts"], c["loc"], c["wts"])
        parity.assert_close("out", out, want, 1e-4)
    assert lib.da_sm100_backward_ws(*(t.data_ptr() for t in ptrs), nbytes - 1, *dims,
                                    capi.dtype_code(dtype), stream) == -6
