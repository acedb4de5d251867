"""Deformable aggregation with operands that do not share a type, and with operands off the vector
kernels' alignment: both are computed as from float32 operands, at the sizes of either backward."""
import pytest
import torch

from tests.test_da_gpu import _random_case

pytestmark = pytest.mark.gpu

NAMES = ("feat", "loc", "wts", "grad_out")
# B, C, A, Pts, G, maps; the second has samples enough for the cell-sorted backward in any type
CASES = [
    (1, 128, 9, 5, 8, [[(30, 176), (4, 4)]]),
    (2, 128, 420, 13, 8, [[(8, 176), (3, 5)], [(20, 20), (4, 9)]]),
]


def _operands(case):
    c = _random_case(case[1] + case[2], *case)
    tables = [torch.from_numpy(c[k]).cuda() for k in ("shapes", "starts")]
    return tables, {k: torch.from_numpy(c[k]).cuda() for k in NAMES}


def _run(tables, t):
    import drivingsdk_b200 as sdk
    leaves = [t[k].detach().requires_grad_() for k in NAMES[:3]]
    out = sdk.deformable_aggregation(leaves[0], *tables, *leaves[1:])
    return (out.detach(), *torch.autograd.grad(out, leaves, t["grad_out"]))


def _agree(got, want):
    """fp32 sums of the same products in another order, then each result rounded to its type."""
    for name, a, b in zip(("out", "grad_feat", "grad_loc", "grad_wts"), got, want):
        unit = torch.finfo(a.dtype).eps
        limit = (1e-4 if name == "grad_loc" else 1e-5) + unit
        assert (a.double() - b.double()).norm() <= limit * b.double().norm(), name


@pytest.mark.parametrize("case", CASES, ids=["few", "sorted"])
@pytest.mark.parametrize("feat", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("narrow", [(), ("wts",), ("loc",)], ids=["feat", "wts", "loc"])
def test_operands_of_different_types(case, feat, narrow):
    tables, t = _operands(case)
    t["feat"] = t["feat"].to(feat)
    t["grad_out"] = t["grad_out"].to(feat)   # autograd hands it over in the output's type
    for k in narrow:
        t[k] = t[k].to(feat)
    want = _run(tables, {k: v.float() for k, v in t.items()})
    got = _run(tables, t)
    assert got[0].dtype == feat and all(g.dtype == t[k].dtype for g, k in zip(got[1:], NAMES))
    _agree(got, want)


@pytest.mark.parametrize("case", CASES, ids=["few", "sorted"])
def test_gradient_of_another_type(case):
    """The extension's own backward takes a float32 gradient of 16-bit features: one that float16
    does not hold, for features and weights small enough that the results are in its range."""
    from drivingsdk_b200 import _C
    tables, t = _operands(case)
    t = {k: v.half() * (1e-4 if k in ("feat", "wts") else 1) for k, v in t.items()}
    go = t["grad_out"].float() * 1e5
    call = lambda f, l, w: _C.npu_deformable_aggregation_backward(f, *tables, l, w, go, f, l, w)  # noqa: E731
    got = call(t["feat"], t["loc"], t["wts"])
    want = call(t["feat"].float(), t["loc"].float(), t["wts"].float())
    _agree([got[0], *got], [want[0], *want])


def _off_by_one_element(t):
    return torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")[1:].view(t.shape).copy_(t)


@pytest.mark.parametrize("case", CASES, ids=["few", "sorted"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("name", NAMES)
def test_contiguous_operands_at_odd_addresses(case, dtype, name):
    tables, t = _operands(case)
    t = {k: v.to(dtype) for k, v in t.items()}
    want = _run(tables, t)
    t[name] = _off_by_one_element(t[name])
    assert t[name].is_contiguous() and t[name].data_ptr() % (2 * t[name].element_size()) != 0
    _agree(_run(tables, t), want)
