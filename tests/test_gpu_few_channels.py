"""Accumulated outer products and products with shared weights of few channels against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from equitorch_b200.ops.batched_sparse_dense_op import indexed_outer_scale_gather, indexed_vecmat_scale_gather

DEV = "cuda:0"


# fewer samples than teams, a block of 128 threads and its remainders, several samples a thread, several chunks; teams of 1 to 256 threads,
# teams that do not divide a block (24 x 24: 36 threads), sizes just outside (68 x 64, 20 columns)
@pytest.mark.parametrize("n", [1, 5, 127, 129, 700, 5003])
@pytest.mark.parametrize("c1,c2", [(4, 4), (16, 16), (24, 24), (16, 32), (64, 32), (64, 64), (68, 64), (20, 20)])
def test_against_float64(n, c1, c2):
    if n * (c1 + c2) > 400_000:
        pytest.skip("large")
    g = torch.Generator().manual_seed(n + c1)
    rows1, rows2, entries, out = 7, 5, 23, 9
    a, b = torch.randn(n, rows1, c1, generator=g).to(DEV), torch.randn(n, rows2, c2, generator=g).to(DEV)
    w = torch.randn(rows2, c1, c2, generator=g).to(DEV)
    i1, i2 = torch.randint(0, rows1, (entries,), generator=g).to(DEV), torch.randint(0, rows2, (entries,), generator=g).to(DEV)
    scale = torch.randn(entries, generator=g).to(DEV)
    seg = torch.tensor([0, 3, 3, 12, 13, 14, 16, 20, 22, 23], device=DEV)                 # one output without entries, one of nine
    place = torch.repeat_interleave(torch.arange(out, device=DEV), seg[1:] - seg[:-1])
    index_out = torch.tensor([4, 0, 8, 10, 2, 3, 7, 1, 6], device=DEV)                    # rows 5 and 9 of the output stay zero

    pair = torch.einsum("nta,ntb->tab", a.double()[:, i1] * scale.double()[:, None], b.double()[:, i2])
    want = torch.zeros(out, c1, c2, dtype=torch.float64, device=DEV).index_add_(0, place, pair)
    got = indexed_outer_scale_gather(a, b, scale, i1, i2, seg, out_accumulated=True, out_size=out)
    # sums of n products a term: 1e-5 of the largest entry is the path's tolerance
    assert float((got.double() - want).abs().max()) <= 1e-5 * float(want.abs().max())

    one = torch.einsum("nta,tab->ntb", a.double()[:, i1] * scale.double()[:, None], w.double()[i2])
    want = torch.zeros(n, 11, c2, dtype=torch.float64, device=DEV).index_add_(1, index_out[place], one)
    got = indexed_vecmat_scale_gather(a, w, scale, i1, i2, seg, index_out=index_out, out_size=11)
    assert float((got.double() - want).abs().max()) <= 1e-5 * float(want.abs().max())


@pytest.mark.parametrize("shift", [1, 2, 4])
def test_operands_off_sixteen_bytes(shift):
    g = torch.Generator().manual_seed(shift)
    n, rows, c = 300, 3, 16
    flat = torch.randn(n * rows * c + 8, generator=g).to(DEV)
    a, w = flat[shift:shift + n * rows * c].view(n, rows, c), torch.randn(rows, c, c, generator=g).to(DEV)
    b = torch.randn(n, rows, c, generator=g).to(DEV)
    got = indexed_vecmat_scale_gather(a, w, out_size=rows)
    want = torch.einsum("nra,rab->nrb", a.double(), w.double())
    assert float((got.double() - want).abs().max()) <= 1e-5 * float(want.abs().max())
    got = indexed_outer_scale_gather(a, b, out_accumulated=True, out_size=rows)
    want = torch.einsum("nra,nrb->rab", a.double(), b.double())
    assert float((got.double() - want).abs().max()) <= 1e-5 * float(want.abs().max())


# two and four samples a thread, the last block of both full of samples or not; 24 input channels keep 32 columns on these kernels
@pytest.mark.parametrize("n", [2000, 4096, 4097, 5003])
@pytest.mark.parametrize("c1,c2", [(16, 16), (24, 32)])
def test_products_of_many_outputs(n, c1, c2):
    g = torch.Generator().manual_seed(n + c2)
    rows, out = 13, 40
    a, w = torch.randn(n, rows, c1, generator=g).to(DEV), torch.randn(rows, c1, c2, generator=g).to(DEV)
    i1, i2 = torch.randint(0, rows, (3 * out,), generator=g).to(DEV), torch.randint(0, rows, (3 * out,), generator=g).to(DEV)
    scale = torch.randn(3 * out, generator=g).to(DEV)
    seg = torch.arange(0, 3 * out + 1, 3, device=DEV)
    got = indexed_vecmat_scale_gather(a, w, scale, i1, i2, seg, out_size=out)
    want = torch.einsum("nta,tab->ntb", a.double()[:, i1] * scale.double()[:, None], w.double()[i2]).view(n, out, 3, c2).sum(2)
    assert float((got.double() - want).abs().max()) <= 1e-5 * float(want.abs().max())


@pytest.mark.parametrize("n,c1,c2", [(450, 64, 64), (1000, 48, 40), (5000, 128, 16), (5000, 8, 128)])
def test_sums_of_one_entry_keep_the_error_of_tiles(n, c1, c2):
    """K additions one after the other of terms of random sign, each rounded by at most half a unit of the partial sum, are off by at
    most 2^-24 sqrt(K / 6) of the norm of the result.  Tiles of 64 x 64 add up their samples and as many chunks as four blocks an SM are, of
    at least 32 samples; the teams of few channels make no longer sums than that."""
    sms = torch.cuda.get_device_properties(DEV).multi_processor_count
    rows = 4
    chunks = min(-(-4 * sms // (rows * -(-c1 // 64) * -(-c2 // 64))), -(-n // 32))
    g = torch.Generator().manual_seed(n)
    a, b = torch.randn(n, rows, c1, generator=g).to(DEV), torch.randn(n, rows, c2, generator=g).to(DEV)
    got = indexed_outer_scale_gather(a, b, out_accumulated=True, out_size=rows)
    want = torch.einsum("nra,nrb->rab", a.double(), b.double())
    assert float((got.double() - want).norm() / want.norm()) <= 2.0 ** -24 * ((chunks + n / chunks) / 6) ** 0.5
