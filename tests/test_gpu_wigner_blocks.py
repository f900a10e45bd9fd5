"""Float32 block kernels of the Wigner-D path (generation, angle gradients, rotation, matrix gradient) against the float64
kernels on the same inputs, where their groups and tiles end: one sample, ragged groups of four, one-row blocks, repeated and
unordered irreps, degree 7, channel counts of one vector up to two tiles, and the forms that stay on the general kernels."""
import pytest
import torch

from equitorch_b200 import nn as enn
from equitorch_b200.irreps import Irreps
from equitorch_b200.ops.wigner_op import block_diagonal, dense_rotation, dense_rotation_grad_matrix

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
# largest difference over largest value: float32 sums of up to 15 (rotation), 64 (matrix gradient), 600 (angles) terms
TOL = 1e-5


def _err(a, b):
    return float((a.double() - b.double()).abs().max()) / max(1e-30, float(b.double().abs().max()))


def _angles(n, gen):
    return [((torch.rand(n, generator=gen) * 2 - 1) * 3.1).to(DEV) for _ in range(3)]


@pytest.mark.parametrize("n", [1, 3, 4, 37, 1025])
@pytest.mark.parametrize("name", ["0e", "1o", "0e+1o+2e", "4x0e+2x1o+2e", "3o+1o+0e+3o", "7o", "0e+1o+2e+3o+4e+5o+6e", "0e+1o+2e+3o+4e+5o+6e+7o"])
def test_generation_and_angle_gradients(name, n):
    ir, gen = Irreps(name), torch.Generator().manual_seed(n)
    angles = _angles(n, gen)
    cot = torch.randn(n, ir.dim, ir.dim, generator=gen).to(DEV)
    results = []
    for dtype in (torch.float32, torch.float64):
        leaves = [a.to(dtype).requires_grad_(True) for a in angles]
        d = enn.WignerD(ir).to(DEV)(*leaves)
        results.append([d.detach(), *torch.autograd.grad(d, leaves, cot.to(dtype))])
    for i, (a, b) in enumerate(zip(*results)):
        if float(b.abs().max()) < 1e-12:                  # a scalar does not depend on the angles
            assert float(a.abs().max()) < 1e-6
        else:
            assert _err(a, b) < TOL, i


@pytest.mark.parametrize("c", [4, 20, 32, 64, 5])
@pytest.mark.parametrize("name,n", [("0e", 9), ("5x0e", 7), ("0e+1o+2e", 130), ("3o+1o+0e+3o", 5), ("0e+1o+2e+3o+4e+5o+6e", 37),
                                    ("0e+1o+2e+3o+4e+5o+6e+7o", 6)])
def test_rotation_and_its_gradients(name, n, c):
    ir, gen = Irreps(name), torch.Generator().manual_seed(n + c)
    mask = torch.zeros(ir.dim, ir.dim)
    at = 0
    for i in ir:
        mask[at:at + i.dim, at:at + i.dim] = 1
        at += i.dim
    m = (torch.randn(n, ir.dim, ir.dim, generator=gen) * mask).to(DEV)
    x, cot = (torch.randn(n, ir.dim, c, generator=gen).to(DEV) for _ in range(2))
    rotate = enn.DenseWignerRotation(ir)
    for transposed in (False, True):
        xa, ma = x.clone().requires_grad_(True), m.clone().requires_grad_(True)
        out = rotate(xa, ma.transpose(-1, -2) if transposed else ma)
        got = [out, *torch.autograd.grad(out, [xa, ma], cot)]
        xd, md, cd = x.double(), m.double(), cot.double()
        t = md.transpose(-1, -2) if transposed else md
        gm = cd @ xd.transpose(-1, -2)
        want = [t @ xd, t.transpose(-1, -2) @ cd, (gm.transpose(-1, -2) if transposed else gm) * mask.to(DEV)]
        for a, b in zip(got, want):
            assert _err(a.detach(), b) < TOL
        assert float((got[2] * (1 - mask.to(DEV))).abs().max()) == 0.0


@pytest.mark.parametrize("name,c", [("109x0e", 4), ("96x0e", 32), ("60x0e+12x1o+2e", 4), ("9x5o", 8), ("64x0e", 128)])
def test_as_many_blocks_as_are_accepted(name, c):
    """Every word of the list of row tiles is in use: the block sizes of the largest matrices that the block kernels take."""
    ir, n, gen = Irreps(name), 5, torch.Generator().manual_seed(c)
    assert block_diagonal(ir, DEV).takes(torch.empty(n, ir.dim, c, device=DEV))
    m = torch.stack([torch.block_diag(*[torch.randn(i.dim, i.dim, generator=gen) for i in ir]) for _ in range(n)]).to(DEV)
    x = torch.randn(n, ir.dim, c, generator=gen).to(DEV)
    for t in (m, m.transpose(-1, -2)):
        assert _err(enn.DenseWignerRotation(ir)(x, t), t.double() @ x.double()) < TOL


def test_what_lies_outside_the_blocks_is_not_read():
    ir = Irreps("0e+1o+2e")
    gen = torch.Generator().manual_seed(2)
    m, x = torch.randn(5, 9, 9, generator=gen).to(DEV), torch.randn(5, 9, 8, generator=gen).to(DEV)
    sizes = [i.dim for i in ir]
    inside = torch.block_diag(*[torch.ones(s, s) for s in sizes]).bool().to(DEV)
    rotate = enn.DenseWignerRotation(ir)
    assert torch.equal(rotate(x, torch.where(inside, m, torch.nan)), rotate(x, torch.where(inside, m, 0.0)))


def test_features_at_an_odd_offset_take_the_general_kernel():
    ir = Irreps("0e+1o+2e")
    gen = torch.Generator().manual_seed(3)
    m = torch.block_diag(*[torch.randn(i.dim, i.dim, generator=gen) for i in ir]).expand(4, 9, 9).contiguous().to(DEV)
    store = torch.randn(4 * 9 * 8 + 1, generator=gen).to(DEV)
    x = store[1:].view(4, 9, 8)
    assert not block_diagonal(ir, x.device).takes(x)
    assert _err(enn.DenseWignerRotation(ir)(x, m), m.double() @ x.double()) < TOL


@pytest.mark.parametrize("name,n,c", [("0e+1o+2e+3o+4e+5o+6e", 3001, 4), ("0e+1o+2e+3o+4e+5o+6e", 1303, 36), ("0e+1o+2e", 40003, 12),
                                      ("9x5o", 701, 8), ("7o", 9002, 64)])
def test_several_images_a_block(name, n, c):
    """More samples than one round of blocks holds, the last image not full; entries outside the blocks stay zero.  A sum of
    c products made in chains of at most c / 4 + 1 multiply-adds with two further additions differs from the exact one by at most
    (c / 4 + 3) eps times the sum of the magnitudes."""
    ir, gen = Irreps(name), torch.Generator().manual_seed(c)
    mask = torch.block_diag(*[torch.ones(i.dim, i.dim) for i in ir]).to(DEV)
    g, x = (torch.randn(n, ir.dim, c, generator=gen).to(DEV) for _ in range(2))
    out = dense_rotation_grad_matrix(g, x, block_diagonal(ir, DEV))
    exact = (g.double() @ x.double().mT) * mask
    most = (g.double().abs() @ x.double().abs().mT) * mask
    assert ((out - exact).abs() <= (c / 4 + 3) * 2.0 ** -24 * most).all()


@pytest.mark.parametrize("name,n,c", [("0e+1o+2e", 301, 12), ("0e+1o", 9001, 4), ("0e+1o+2e", 40003, 8)])
def test_matrix_gradient_of_few_channels(name, n, c):
    """Few samples, blocks too small for one lane an item, and one lane an item, whose chains of c / 2 multiply-adds meet in one addition."""
    ir, gen = Irreps(name), torch.Generator().manual_seed(c)
    mask = torch.block_diag(*[torch.ones(i.dim, i.dim) for i in ir]).to(DEV)
    g, x = (torch.randn(n, ir.dim, c, generator=gen).to(DEV) for _ in range(2))
    out = dense_rotation_grad_matrix(g, x, block_diagonal(ir, DEV))
    exact = (g.double() @ x.double().mT) * mask
    most = (g.double().abs() @ x.double().abs().mT) * mask
    assert ((out - exact).abs() <= max(c / 4 + 3, c / 2 + 1) * 2.0 ** -24 * most).all()


@pytest.mark.parametrize("name,n,c", [("0e+1o+2e", 30011, 8), ("7o", 3003, 12), ("5x0e", 9001, 4), ("0e+1o+2e+3o+4e+5o", 2501, 64)])
@pytest.mark.parametrize("skip", [0, 1, 3])
def test_several_passes_of_whole_matrices(name, n, c, skip):
    """More samples than one round of blocks holds, the matrices beginning at any float.  A chain of at most 15 multiply-adds
    differs from the exact sum by at most 15 eps times the sum of the magnitudes."""
    ir, gen = Irreps(name), torch.Generator().manual_seed(c)
    mask = torch.block_diag(*[torch.ones(i.dim, i.dim) for i in ir]).to(DEV)
    m = torch.randn(n * ir.dim ** 2 + skip, generator=gen).to(DEV)[skip:].view(n, ir.dim, ir.dim)
    x = torch.randn(n, ir.dim, c, generator=gen).to(DEV)
    for transposed in (False, True):
        out = dense_rotation(m, x, transposed, block_diagonal(ir, DEV))
        blocks = (m * mask).double()
        blocks = blocks.mT if transposed else blocks
        assert ((out - blocks @ x.double()).abs() <= 15 * 2.0 ** -24 * (blocks.abs() @ x.double().abs())).all()


def test_operands_of_more_than_eight_hundred_megabytes_by_the_list():
    for skip in (0, 1, 3):
        test_several_passes_of_whole_matrices("0e+1o+2e+3o+4e+5o", 34003, 64, skip)
