"""The counting sort behind the sorted backward, where its counters are kept in another way or its
samples end up elsewhere: clusters that merge, split or do not share their counters, sorted numbers
staged in shared memory or not, more cells than one pass holds, points per query that do not divide
the CTA's threads. Checked through the operator, against the oracle."""
import pytest
import torch

from drivingsdk_b200 import capi, workloads
from tests import parity

pytestmark = pytest.mark.gpu

# B, Q, H, D, levels, P, loc_range
CASES = {
    "merged": (1, 3000, 1, 8, ((40, 50),), 8, (-0.1, 1.1)),            # 11 samples per cell
    "alone-staged": (1, 3000, 1, 8, ((9, 13),), 8, (-0.1, 1.1)),       # 171
    "split": (1, 3000, 1, 8, ((150, 200), (60, 70)), 7, (-0.1, 1.1)),  # below one
    "split-two-passes": (1, 900, 1, 4, ((450, 480),), 7, (0.0, 1.0)),  # 216931 cells
    "alone": (8, 5900, 37, 4, ((6, 6),), 5, (-0.1, 1.1)),              # 29500 samples per map: no room
    "all-dropped": (1, 400, 2, 8, ((5, 6), (3, 4)), 3, (1.5, 2.5)),
}


@pytest.mark.parametrize("case", CASES)
def test_sorted_backward_of_every_kind_of_counters(case):
    B, Q, H, D, levels, P, loc_range = CASES[case]
    inp = workloads.make_inputs(workloads.Workload("sort", B, Q, H, D, levels, P, loc_range, seed=11), torch.float32)
    dev = parity.to_device(inp, torch.float32)
    old = capi.load().msda_sm100_tune(capi.TUNE_SORT, 2)
    try:
        parity.compare_all(inp, parity.run_python_api(dev), torch.float32)
    finally:
        capi.load().msda_sm100_tune(capi.TUNE_SORT, old)
    assert capi.load().msda_sm100_device_status(1) == 0
