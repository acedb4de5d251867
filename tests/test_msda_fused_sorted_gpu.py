"""The fused operator's backward over cell-sorted samples: against its unsorted form (the same locations,
weights and cells, sums in another order) with items of one and of several tasks, tasks of one sample, idle
lanes, levels of one pixel, samples outside; and against the float64 composition where the rule takes it."""
import pytest
import torch

from drivingsdk_b200 import capi, workloads
from tests import parity, test_msda_fused_gpu
from tests.test_msda_fused_gpu import _inputs, _run

pytestmark = pytest.mark.gpu

CASES = {   # B, Q, H, D, levels, P
    "lp1": (1, 129, 2, 128, ((6, 6),), 1),
    "lp4": (2, 333, 8, 32, ((40, 40),), 4),
    "lp15": (1, 301, 3, 24, ((9, 7), (5, 4), (1, 1)), 5),
    "lp16": (1, 300, 8, 64, ((32, 32), (16, 16), (8, 8), (4, 4)), 4),
    "lp32": (2, 200, 4, 16, ((29, 50), (15, 25), (8, 13), (4, 7)), 8),
    "few": (1, 1, 1, 4, ((3, 2),), 3),
    "d256": (1, 150, 2, 256, ((12, 10), (6, 5)), 4),
    "d100": (1, 150, 2, 100, ((12, 10), (6, 5)), 4),
}


def _launches(dtype, sort):   # forward, backward in one kernel or four, conversion of 16-bit sums
    return 1 + (4 if sort else 1) + (0 if dtype == torch.float32 else 1)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("case", CASES)
def test_sorted_equals_unsorted(case, dtype):
    B, Q, H, D, levels, P = CASES[case]
    inp = _inputs(workloads.Workload("fs", B, Q, H, D, levels, P, (0, 1), 3), dtype, seed=Q)
    results = []
    for sort in (0, 2):
        old = capi.load().msda_sm100_tune(capi.TUNE_SORT, sort)
        before = capi.load().msda_sm100_launch_count()
        try:
            results.append(_run(inp, dtype))
        finally:
            capi.load().msda_sm100_tune(capi.TUNE_SORT, old)
        assert capi.load().msda_sm100_launch_count() - before == _launches(dtype, sort != 0)
    # sums of up to some hundred products in another order; 16-bit results may round to a neighbour
    tol = 2e-5 if dtype == torch.float32 else parity.TOL[dtype]
    for name, a, b in zip(("out", "grad_value", "grad_ref", "grad_off", "grad_logits"), *results):
        scale = max(1.0, a.float().abs().max().item())
        assert (a.float() - b.float()).abs().max().item() <= tol * scale, name
    assert capi.load().msda_sm100_device_status(1) == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_sorted_by_the_rule_matches_float64_composition(dtype):
    w = workloads.Workload("fs", 1, 2100, 8, 128, ((32, 32), (16, 16), (8, 8), (4, 4)), 4, (0, 1), 3)   # 0.27 M samples
    before = capi.load().msda_sm100_launch_count()
    test_msda_fused_gpu.test_fused_matches_float64_composition("sorted", w, dtype)
    assert capi.load().msda_sm100_launch_count() - before == _launches(dtype, True)
