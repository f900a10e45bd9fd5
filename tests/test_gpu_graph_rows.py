"""Rows of nodes and edges: gather, segment sum and their adjoints against float64 indexing, where their units, runs of rows
and segments end."""
import pytest
import torch

from equitorch_b200.ops.graph_ops import _scatter_add_rows_raw, gather_rows, segment_sum

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float64])
def test_the_adjoint_of_the_gather_is_deterministic_on_request(dtype):
    g = torch.Generator(device=DEV).manual_seed(0)
    x = torch.randn(7, 33, generator=g, device=DEV).to(dtype).requires_grad_(True)
    index = torch.randint(0, 7, (40000,), generator=g, device=DEV)
    cot = torch.randn(40000, 33, generator=g, device=DEV).to(dtype)
    before = torch.are_deterministic_algorithms_enabled()
    torch.use_deterministic_algorithms(True)
    try:
        runs = [torch.autograd.grad(gather_rows(x, index), x, cot)[0] for _ in range(8)]
    finally:
        torch.use_deterministic_algorithms(before)
    assert all(torch.equal(r, runs[0]) for r in runs)
    want = torch.zeros(7, 33, device=DEV, dtype=torch.float64).index_add_(0, index, cot.double())
    # sums of 5700 terms: in order in float32 1e-5 of the largest, in bfloat16 storage one rounding per addition
    assert float((runs[0].double() - want).abs().max() / want.abs().max()) < {torch.float32: 1e-5, torch.float64: 1e-12}.get(dtype, 1.0)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_derivatives_of_the_adjoints(dtype):
    """A gradient that is itself differentiated, for the gather and the segment sum."""
    g = torch.Generator(device=DEV).manual_seed(1)
    x = torch.randn(11, 5, generator=g, device=DEV, dtype=dtype).requires_grad_(True)
    index = torch.randint(0, 11, (40,), generator=g, device=DEV)
    ptr = torch.tensor([2, 2, 9, 30, 36], device=DEV)

    def second(fn):
        out = fn(x)
        (first,) = torch.autograd.grad((out ** 3).sum(), x, create_graph=True)
        return [out, first, *torch.autograd.grad((first ** 2).sum(), x)]

    def plain(t):
        rows = t[index]
        return torch.stack([rows[a:b].sum(0) for a, b in zip(ptr[:-1].tolist(), ptr[1:].tolist())])
    for a, b in zip(second(lambda t: segment_sum(gather_rows(t, index), ptr)), second(plain)):
        assert float((a - b).abs().max() / b.abs().max()) < (1e-5 if dtype == torch.float32 else 1e-12)


@pytest.mark.parametrize("width,dtype", [(64, torch.float32), (3, torch.float32), (1, torch.float32), (45, torch.bfloat16),
                                         (480, torch.bfloat16), (6, torch.float64), (1028, torch.float32)])
@pytest.mark.parametrize("bounds", [[0, 0], [0, 1], [5, 12], [0, 15, 16, 17, 64, 64, 64, 200], [3, 3, 3, 40, 41], [0, 200], [0, 16, 32, 48, 200],
                                    [0] * 40 + list(range(0, 100, 3)) + [100] * 70 + [190]])
def test_adjoint_of_the_segment_sum(bounds, width, dtype):
    """Few long and many short segments; segments that end at, before and after the runs of 16 rows, empty ones, and rows before
    the first and after the last."""
    g = torch.Generator(device=DEV).manual_seed(width)
    rows, ptr = 200, torch.tensor(bounds, device=DEV)
    x = torch.randn(rows, width, generator=g, device=DEV).to(dtype).requires_grad_(True)
    cot = torch.randn(len(bounds) - 1, width, generator=g, device=DEV).to(dtype)
    (got,) = torch.autograd.grad(segment_sum(x, ptr), x, cot)
    want = torch.zeros_like(got)
    for d, (a, b) in enumerate(zip(bounds, bounds[1:])):
        want[a:b] = cot[d]
    assert torch.equal(got, want)


def _rows(g, rows, width, dtype, offset):
    """Rows whose first element lies ``offset`` elements behind a 16-byte boundary."""
    return torch.randn(rows * width + offset, generator=g, device=DEV).to(dtype)[offset:].view(rows, width)


@pytest.mark.parametrize("offset", [0, 1, 4])
@pytest.mark.parametrize("width,dtype", [(64, torch.float32), (3, torch.float32), (1, torch.float32), (6, torch.float32), (1028, torch.float32),
                                         (45, torch.bfloat16), (480, torch.bfloat16), (12, torch.bfloat16), (1, torch.bfloat16),
                                         (6, torch.float64), (5, torch.float64)])
def test_gather_sum_and_the_adjoint_of_the_gather(width, dtype, offset):
    """Units of 16 bytes, of four elements and of one; rows off the 16-byte grid; segments that are empty, shorter and longer than
    the four rows in flight; a permutation of the rows."""
    g = torch.Generator(device=DEV).manual_seed(width + offset)
    x = _rows(g, 57, width, dtype, offset)
    index = torch.randint(0, 57, (301,), generator=g, device=DEV)
    leaf = x.detach().requires_grad_(True)
    picked = gather_rows(leaf, index)
    assert torch.equal(picked, x[index])
    # sums of up to 12 (adjoint), 240 (segments) terms of both signs: float32 1e-6 of the largest, bfloat16 the rounding of the result
    tol = {torch.float32: 1e-5, torch.bfloat16: 2.0 ** -8, torch.float64: 1e-13}[dtype]
    cot = _rows(g, 301, width, dtype, offset)
    (got,) = torch.autograd.grad(picked, leaf, cot)
    want = torch.zeros(57, width, device=DEV, dtype=torch.float64).index_add_(0, index, cot.double())
    assert got.dtype == dtype and float((got.double() - want).abs().max()) <= tol * float(want.abs().max())
    bounds = [0, 0, 1, 4, 9, 249, 249, 290]
    ptr, perm = torch.tensor(bounds, device=DEV), torch.randperm(301, generator=g, device=DEV)
    for order in (None, perm):
        got = segment_sum(cot, ptr) if order is None else segment_sum(cot, ptr, order)
        rows = cot.double() if order is None else cot.double()[order]
        want = torch.stack([rows[a:b].sum(0) for a, b in zip(bounds, bounds[1:])])
        assert got.dtype == dtype and float((got.double() - want).abs().max()) <= tol * float(want.abs().max())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rows_added_outside_the_result_are_skipped(dtype):
    g = torch.Generator(device=DEV).manual_seed(2)
    rows, index = torch.randn(6, 8, generator=g, device=DEV).to(dtype), torch.tensor([0, -1, 2, 3, 1 << 40, 0], device=DEV)
    want = torch.zeros(3, 8, device=DEV).index_add_(0, index[[0, 2, 5]], rows[[0, 2, 5]].float())
    assert torch.equal(_scatter_add_rows_raw(rows, index, 3), want.to(dtype))
    assert torch.equal(_scatter_add_rows_raw(rows[:0], index[:0], 3), torch.zeros(3, 8, device=DEV, dtype=dtype))
    assert _scatter_add_rows_raw(rows[:0], index[:0], 0).shape == (0, 8)
