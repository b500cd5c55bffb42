"""The parameter gradients of an instance of one tile (at most 128 columns) have one order of
summation: the same bits on every call, also beside another stream's work, which changes the order
in which a block's warps end."""
import importlib

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kx,ix,il", [(8, 16, 8), (16, 16, 8), (16, 43, 2), (7, 8, 5)])
def test_repeated_calls_give_the_same_bits(kx, ix, il):
    import torch
    pkg = importlib.import_module("jax-gcm_b200")
    make = lambda seed, *shape: pkg.instance_to_device(
        pkg.synthetic.land_instance(seed, *shape), "cuda")
    phys = pkg.SpeedyPhysics(diagnostics=False)
    cot = lambda *shape: pkg.PhysicsTendency(*(torch.randn(shape, device="cuda")
                                               for _ in range(4)))
    one, ct = make(kx + ix, ix, il, kx), cot(kx, ix, il)
    beside, ct2 = make(5, 128, 64, 16), cot(16, 128, 64)
    first = pkg.adjoint.vjp(phys, *one, ct)[1]
    torch.cuda.synchronize()
    assert first.abs().max() > 0
    stream, got = torch.cuda.Stream(), []
    for _ in range(1000):
        with torch.cuda.stream(stream):
            pkg.adjoint.vjp(phys, *beside, ct2)
        got.append(pkg.adjoint.vjp(phys, *one, ct)[1])
    torch.cuda.synchronize()
    assert all(torch.equal(g, first) for g in got)
