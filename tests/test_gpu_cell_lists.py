"""Neighbour lists kept between the search and the edge pass against the path that searches twice (bit-exact) and the
brute-force oracle: one and two points, targets without neighbours, all points in one cell, more neighbours than a row keeps,
blocks of 32 targets and passes of 128 edges that end raggedly, graphs in any order and without points."""
import pytest
import torch

from equitorch_b200 import _lib
from equitorch_b200.ops import featurize_op as fop
from oracle import featurize as ofe

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("l_max,basis", [(None, 0), (0, 3), (3, 8), (4, 1)])
@pytest.mark.parametrize("n,box,r,cap,loop,graphs", [(2, 0.1, 0.5, 4, False, 1), (1, 1.0, 0.5, 4, True, 1), (33, 0.1, 0.5, 64, False, 1),
                                                     (300, 1.0, 2.0, 7, False, 1), (1000, 40.0, 1.0, 32, False, 1),
                                                     (4097, 12.0, 1.3, 48, True, 1), (700, 3.0, 0.9, 600, False, 5)])
def test_lists_equal_the_second_search_and_the_oracle(monkeypatch, n, box, r, cap, loop, graphs, l_max, basis):
    g = torch.Generator().manual_seed(n + cap)
    pos = torch.rand(n, 3, generator=g) * box
    batch = torch.randint(0, graphs, (n,), generator=g) * 2 if graphs > 1 else None
    kw = dict(loop=loop, max_num_neighbors=cap, with_length=True, l_max=l_max, cutoff="polynomial", cutoff_r_max=r)
    if basis:
        kw.update(bessel_weights=torch.arange(1, basis + 1, device=DEV) * torch.pi, bessel_r_max=r)
    args = (pos.to(DEV), r, None if batch is None else batch.to(DEV))
    new = fop.radius_graph_features(*args, **kw)
    monkeypatch.setattr(fop, "MAX_LIST_ENTRIES", 0)
    old = fop.radius_graph_features(*args, **kw)
    for a, b in zip(new, old):
        assert (a is None) == (b is None)
        if a is not None:
            assert a.shape == b.shape and torch.equal(a.nan_to_num(7.0), b.nan_to_num(7.0))      # sin(0) / 0 with loops
    src, dst = ofe.radius_graph(pos, r, batch, loop, cap)
    assert torch.equal(new.src.cpu(), src) and torch.equal(new.dst.cpu(), dst)


def test_too_many_candidates_are_refused_and_the_next_call_is_not():
    pos = torch.rand(600, 3, device=DEV) * 0.1
    for _ in range(2):
        with pytest.raises(_lib.EqtError):
            fop.radius_graph_features(pos, 1.0)
    assert fop.radius_graph_features(pos[:500], 1.0).src.numel() == 500 * 32
