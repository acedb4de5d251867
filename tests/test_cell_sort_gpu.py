"""The counting sort behind the sorted backward, where its counters are kept in another way or its
samples end up elsewhere: clusters that merge, split or do not share their counters, sorted numbers
staged in shared memory or not, more cells than one pass holds, points per query that do not divide
the CTA's threads. Checked through the operator, against the oracle."""
import pytest
import torch

from drivingsdk_b200 import capi, workloads
from tests import parity

pytestmark = pytest.mark.gpu

# B, Q, H, D, levels, P, loc_range, and how each level's map is sorted on 148 SMs (tests/test_sort_choice.py
# asks the library): CTAs, counters, sample numbers staged, the larger shared memory
SPLIT, MERGED, ALONE = range(3)
CASES = {
    "merged": (1, 3000, 1, 8, ((40, 50),), 8, (-0.1, 1.1),             # 11 samples per cell
               [(8, MERGED, False, False)]),
    "alone-staged": (1, 3000, 1, 8, ((9, 13),), 8, (-0.1, 1.1),        # 171, 21 in each CTA
                     [(8, ALONE, True, False)]),
    "split": (1, 3000, 1, 8, ((150, 200), (60, 70)), 7, (-0.1, 1.1),   # below one; below five
              [(8, SPLIT, False, False), (8, MERGED, False, False)]),
    "split-two-passes": (1, 3000, 1, 4, ((450, 480),), 7, (0.0, 1.0),  # 216931 cells, 196608 in a pass
                         [(8, SPLIT, False, False)]),
    "nine-passes": (1, 900, 1, 4, ((450, 480),), 7, (0.0, 1.0),        # ... or 24576, by one CTA
                    [(1, ALONE, False, False)]),
    "alone": (8, 5900, 37, 4, ((6, 6),), 5, (-0.1, 1.1),               # 29500 samples per map: no room
              [(1, ALONE, False, False)]),
    "large-room": (1, 29750, 1, 4, ((9, 13),), 7, (-0.1, 1.1),         # 26032 samples in each CTA
                   [(8, ALONE, True, True)]),
    "all-dropped": (1, 400, 2, 8, ((5, 6), (3, 4)), 3, (1.5, 2.5), 2 * [(1, ALONE, True, False)]),
}


@pytest.mark.parametrize("case", CASES)
def test_sorted_backward_of_every_kind_of_counters(case):
    B, Q, H, D, levels, P, loc_range, _ = CASES[case]
    inp = workloads.make_inputs(workloads.Workload("sort", B, Q, H, D, levels, P, loc_range, seed=11), torch.float32)
    dev = parity.to_device(inp, torch.float32)
    old = capi.load().msda_sm100_tune(capi.TUNE_SORT, 2)
    try:
        parity.compare_all(inp, parity.run_python_api(dev), torch.float32)
    finally:
        capi.load().msda_sm100_tune(capi.TUNE_SORT, old)
    assert capi.load().msda_sm100_device_status(1) == 0
    assert torch.cuda.get_device_properties(0).multi_processor_count == 148   # what the forms are stated for
