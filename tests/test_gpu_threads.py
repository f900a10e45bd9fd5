"""Host threads on one device whose launches of one kernel need different amounts of shared memory."""
import threading

import pytest
import torch

from equitorch_b200 import nn as enn
from equitorch_b200.irreps import Irreps

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _layers(c):
    ir = "0e+1o+2e+3o"
    layer = enn.SO3Linear(ir, ir, ir, c, c, internal_weights=False, feature_mode="uu").to(DEV)
    x, y = torch.randn(40, 16, c, device=DEV), torch.randn(40, 16, device=DEV)
    w = torch.randn(*layer.weight_shape, device=DEV)
    leaves = [t.requires_grad_(True) for t in (x, y, w)]
    return lambda: torch.autograd.grad(layer(*leaves).sum(), leaves)


def _rotations(l_max):
    ir = Irreps((0, l_max))
    wigner, rotate = enn.WignerD(ir).to(DEV), enn.DenseWignerRotation(ir)
    angles = [torch.rand(9, device=DEV).requires_grad_(True) for _ in range(3)]
    x = torch.randn(9, ir.dim, 64, device=DEV)
    return lambda: torch.autograd.grad(rotate(x, wigner(*angles)).sum(), angles)


@pytest.mark.parametrize("make,sizes", [(_layers, (4, 64, 128)), (_rotations, (2, 4, 6))])
def test_threads_with_launches_of_different_size(make, sizes):
    calls, errors = [make(s) for s in sizes], []
    want = [call() for call in calls]

    def work(call, ref):
        try:
            for _ in range(400):
                got = call()
            assert all(torch.allclose(a, b, rtol=1e-4, atol=1e-4 * float(b.abs().max())) for a, b in zip(got, ref))
        except Exception as e:                                   # noqa: BLE001 - handed to the main thread
            errors.append(e)
    threads = [threading.Thread(target=work, args=pair) for pair in zip(calls, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
