"""Which calls the backward over cell-sorted samples takes: the size of the workspace says it. Calls on either
side of the lines, at widths that fill their lanes and widths that do not; 16-bit rows of 8 bytes, which the
unsorted kernel takes one channel at a time, are sorted from 0.1 M samples on. And how the sorts of the GPU
tests divide their work, so that a change of the rules cannot move a test to another path unseen."""
import pytest

from drivingsdk_b200 import capi
from tests.test_cell_sort_gpu import CASES as SORTS

# operator, type, B, K, H, D, L, Q, P, sorted
CALLS = [
    ("msda", "bf16", 4, 165, 4, 4, 2, 15382, 2, True),          # 0.98 M, 373 per cell: 58 us against 488
    ("msda", "bf16", 1, 540, 8, 4, 1, 30486, 3, True),          # 0.73 M, 169: 65 against 415
    ("msda", "bf16", 1, 6, 2, 12, 1, 8000, 4, False),           # 64 K samples: two launches more
    ("msda", "f32", 1, 128, 2, 4, 1, 57564, 4, True),           # 0.46 M, 1799: 83 against 283
    ("msda", "bf16", 2, 806, 1, 16, 3, 20730, 5, True),         # 0.62 M, 386: 56 against 128
    ("msda", "f32", 6, 167, 8, 4, 4, 640, 4, False),             # 0.49 M on few, narrow rows: 26 against 38
    ("msda", "f32", 1, 30825, 8, 32, 4, 2500, 8, False),        # 0.64 M, 2.6
    ("msda", "f32", 2, 17821, 8, 32, 4, 17821, 4, True),        # an encoder
    ("msda", "f32", 6, 30825, 8, 32, 4, 2500, 8, False),        # spatial cross-attention: 2.6 per cell
    ("msda", "bf16", 6, 30825, 8, 32, 4, 2500, 8, True),
    ("msda", "f32", 7, 3000, 8, 24, 3, 2500, 4, True),          # 1.68 M, 10
    ("msda", "bf16", 2, 85000, 4, 8, 3, 37000, 8, False),       # 7.1 M, 10 per cell, 8 channels: 365 against 464
    ("msda", "bf16", 3, 4165, 4, 80, 1, 15000, 1, True),        # 0.18 M, 3.6: 83 against 132
    ("fused", "f32", 3, 1008, 1, 96, 1, 9450, 4, False),        # 0.11 M, 37: 60 against 75
    ("msda", "bf16", 2, 10000, 8, 48, 4, 1500, 4, False),       # 0.38 M, 2.4
    ("msda", "bf16", 2, 2000, 8, 48, 4, 1500, 4, True),         # 0.38 M, 12
    ("fused", "f32", 6, 30825, 8, 32, 4, 2500, 8, False),
    ("fused", "f32", 2, 2000, 8, 64, 4, 4000, 4, True),
    ("fused", "bf16", 2, 100, 8, 16, 1, 40000, 4, False),       # two more kernels cost what the sort gains
    ("fused", "bf16", 2, 100, 8, 12, 1, 40000, 4, True),
    ("gka", "f32", 24, 375, 4, 64, 1, 7156, 15, True),
    ("gka", "f32", 24, 375, 4, 64, 1, 300, 15, False),
]


@pytest.mark.parametrize("call", CALLS, ids=[f"{c[0]}-{c[1]}-d{c[5]}q{c[7]}" for c in CALLS])
def test_workspace_says_whether_a_call_is_sorted(call):
    op, dtype, B, K, H, D, L, Q, P, sort = call
    lib = capi.load()
    code = {"f32": capi.F32, "bf16": capi.BF16}[dtype]
    size = {"msda": lib.msda_sm100_backward_sorted_workspace_bytes,
            "fused": lib.msda_sm100_fused_backward_sorted_workspace_bytes,
            "gka": lib.gka_sm100_backward_sorted_workspace_bytes}[op](B, K, H, D, L, Q, P, code)
    assert (size > lib.msda_sm100_backward_workspace_bytes(B, K, H, D, code)) == sort


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("D", [4, 16, 24, 32, 48, 64, 96, 128, 192, 256])
def test_more_samples_never_leave_the_sorted_form(D, dtype):
    lib, code = capi.load(), {"f32": capi.F32, "bf16": capi.BF16}[dtype]
    for size in (lib.msda_sm100_backward_sorted_workspace_bytes, lib.msda_sm100_fused_backward_sorted_workspace_bytes,
                 lib.gka_sm100_backward_sorted_workspace_bytes):
        chosen = [size(2, 3000, 8, D, 4, Q, 4, code) > lib.msda_sm100_backward_workspace_bytes(2, 3000, 8, D, code)
                  for Q in (100, 390, 400, 1000, 2000, 4000, 8000, 20000, 50000)]
        assert chosen == sorted(chosen)


@pytest.mark.parametrize("case", SORTS)
def test_sorts_take_the_form_they_are_tested_for(case):
    B, Q, H, _, levels, P, _, forms = SORTS[case]
    K, L = sum(h * w for h, w in levels), len(levels)
    for (h, w), (parts, kept, staged, large) in zip(levels, forms):
        got = capi.load().msda_sm100_sort_form(B * H * L, Q * P, K // L, 2 * (K + 1), (h + 1) * (w + 1), 148)
        assert (got & 15, got >> 4 & 3, bool(got & 64), bool(got & 128)) == (parts, kept, staged, large)
