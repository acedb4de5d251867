"""Rows of a number of 16-byte pieces that is not a power of two (heads of 24, 40, 48 ... channels),
whose last lanes have no piece of their own, against the oracle: forward, backward, fused."""
import pytest
import torch

from drivingsdk_b200 import capi, workloads
from tests import parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D", [24, 40, 48, 72, 160, 200])
def test_rows_that_leave_lanes_idle(D, dtype):
    w = workloads.Workload("rows", 2, 61, 3, D, ((9, 12), (5, 6), (1, 2)), 3, (-0.1, 1.1), seed=D)
    inp = workloads.make_inputs(w, dtype)
    dev = parity.to_device(inp, dtype)
    old = capi.load().msda_sm100_tune(capi.TUNE_SORT, 0)
    try:
        parity.compare_all(inp, parity.run_python_api(dev), dtype)
        if dtype == torch.float32:
            parity.compare_all(inp, parity.run_c_abi(dev, dtype, workspace=False), dtype)
    finally:
        capi.load().msda_sm100_tune(capi.TUNE_SORT, old)
    assert capi.load().msda_sm100_device_status(1) == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D,L,P", [(32, 1, 1), (32, 1, 3), (32, 1, 4), (16, 2, 4), (8, 3, 5), (64, 1, 2),
                                   (128, 1, 1), (24, 1, 4)])
def test_tasks_of_few_rows(D, L, P, dtype):
    """Several tasks per warp, one per group of lanes: task counts that leave groups without one,
    tasks that share several groups, a last item that is not full."""
    levels = ((7, 9), (4, 5), (2, 2))[:L]
    w = workloads.Workload("few", 1, 37, 3, D, levels, P, (-0.2, 1.2), seed=D + P)
    inp = workloads.make_inputs(w, dtype)
    parity.compare_all(inp, parity.run_python_api(parity.to_device(inp, dtype)), dtype)
