"""The backward over cell-sorted samples (MSDA_TUNE_SORT = 2 takes it at any size) against the
oracle, at the sizes where its tiling can go wrong: rows of every lane layout and rows that leave
lanes idle, runs shorter and longer than a stream, one pixel, samples that all share one cell,
levels larger than one CTA's counters."""
import numpy as np
import pytest
import torch

from drivingsdk_b200 import capi, workloads
from oracle import msda_oracle
from tests import parity

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def always_sort():
    old = capi.load().msda_sm100_tune(capi.TUNE_SORT, 2)
    yield
    capi.load().msda_sm100_tune(capi.TUNE_SORT, old)


CASES = [
    # B, Q, H, D, levels, P, loc_range
    (1, 7, 1, 4, ((1, 1),), 1, (-0.5, 1.5)),
    (2, 130, 3, 8, ((5, 3), (1, 2)), 3, (-0.2, 1.2)),
    (1, 333, 2, 16, ((9, 7), (4, 4)), 5, (-0.1, 1.1)),
    (2, 257, 4, 24, ((16, 12), (8, 6)), 4, (-0.1, 1.1)),
    (1, 200, 2, 32, ((12, 9),), 4, (0.49, 0.51)),          # everything in one or two cells
    (1, 600, 2, 48, ((6, 10), (3, 5), (2, 3)), 4, (-0.1, 1.1)),
    (3, 70, 2, 64, ((20, 20),), 7, (-0.1, 1.1)),
    (1, 150, 3, 128, ((10, 14), (5, 7)), 4, (-0.1, 1.1)),
    (1, 90, 2, 256, ((7, 9),), 8, (-0.1, 1.1)),
    (1, 120, 2, 256, ((40, 60), (20, 30)), 4, (-0.1, 1.1)),   # some dot products in double
    (1, 100, 2, 192, ((40, 60),), 4, (-0.1, 1.1)),
    (1, 150, 3, 96, ((10, 14), (5, 7)), 4, (-0.1, 1.1)),      # under 40 samples per pixel
    (1, 400, 2, 96, ((6, 7), (3, 4)), 4, (-0.1, 1.1)),        # more
    (1, 900, 1, 32, ((210, 240), (2, 2)), 2, (0.0, 1.0)),  # 50851 cells: more than one CTA holds
]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("case", CASES, ids=[f"d{c[3]}q{c[1]}" for c in CASES])
def test_sorted_backward_matches_the_oracle(case, dtype):
    B, Q, H, D, levels, P, loc_range = case
    w = workloads.Workload("sorted", B, Q, H, D, levels, P, loc_range, seed=7 + D + Q)
    inp = workloads.make_inputs(w, dtype)
    dev = parity.to_device(inp, dtype)
    parity.compare_all(inp, parity.run_python_api(dev), dtype)
    assert capi.load().msda_sm100_device_status(1) == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D", [8, 32, 64, 128, 256])
def test_sorted_nearest_pixel_backward(D, dtype):
    import drivingsdk_b200 as sdk
    rng = np.random.default_rng(D)
    B, Q, H, P, hw = 2, 210, 3, 7, (5, 8)
    rnd = lambda a: torch.from_numpy(a.astype(np.float32)).to(dtype)  # noqa: E731
    value, attn = rnd(rng.random((B, 40, H, D))), rnd(rng.random((B, Q, H, 1, P)))
    loc = rnd(np.stack([rng.integers(-2, 10, (B, Q, H, 1, P)), rng.integers(-2, 7, (B, Q, H, 1, P))], -1))
    go = rnd(rng.random((B, Q, H * D)))
    shapes, starts = np.array([hw], np.int32), np.array([0], np.int32)
    v, a = value.cuda().requires_grad_(), attn.cuda().requires_grad_()
    out = sdk.geometric_kernel_attention(v, torch.from_numpy(shapes).cuda(),
                                         torch.from_numpy(starts).cuda(), loc.cuda(), a)
    gv, ga = torch.autograd.grad(out, (v, a), go.cuda())
    n = lambda t: t.float().numpy()  # noqa: E731
    want_gv, want_ga = msda_oracle.gka_backward(n(value), shapes, starts, n(loc), n(attn), n(go))
    tol = parity.TOL[dtype]
    if dtype != torch.float32:
        want_gv, want_ga = (torch.from_numpy(x).to(dtype).double().numpy() for x in (want_gv, want_ga))
    parity.assert_close("grad_value", gv, want_gv, tol)
    parity.assert_close("grad_attn", ga, want_ga, tol)
