"""The rollout's vector updates against the multi-tensor operations they stand for, bit for bit:
one launch for the forward step, one for the reverse; plane sizes that are not a multiple of four,
planes off their 16-byte alignment, and what the kernels leave to the general path."""
import importlib

import pytest

pytestmark = pytest.mark.gpu
EVOLVED = ("u_wind", "v_wind", "temperature", "specific_humidity")


@pytest.fixture(scope="module")
def pkg():
    return importlib.import_module("jax-gcm_b200")


def _planes(shape, seed, off=0):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n = 1
    for s in shape:
        n *= s
    new = lambda: torch.randn(n + off, generator=gen, device="cuda")[off:].view(shape)
    return [new() for _ in range(4)]


@pytest.mark.parametrize("shape,off", [((8, 64, 32), 0), ((7, 5, 3), 0), ((16, 1, 1), 0),
                                       ((7, 1, 1), 0), ((8, 16, 4), 1), ((16, 320, 160), 0)])
def test_updates_match_multi_tensor_operations(pkg, shape, off):
    import torch
    calls, dt = pkg._lib.calls(), 1800.0
    x, f = _planes(shape, 1, off), _planes(shape, 2, off)
    rc, got = calls.rollout_step(x, f, dt)
    assert rc == 0
    for a, b in zip(got, torch._foreach_add(x, f, alpha=dt)):
        assert torch.equal(a, b)
    g = pkg.PhysicsState(*_planes(shape, 3, off), _planes(shape, 4)[0], _planes(shape[1:], 5)[0])
    gp = torch.randn(12, device="cuda")
    phi, psa, par = _planes(shape, 6)[0], _planes(shape[1:], 7)[0], torch.randn(12, device="cuda")
    want = torch._foreach_add([phi, psa, par], [g.geopotential, g.normalized_surface_pressure, gp])
    rc, out = calls.rollout_reverse(x, g, gp, phi, psa, par, dt)
    assert rc == 0
    xb = list(torch._foreach_add(x, [getattr(g, k) for k in EVOLVED]))
    for a, b in zip(out, xb + list(torch._foreach_mul(xb, dt))):
        assert torch.equal(a, b)
    for a, b in zip((phi, psa, par), want):
        assert torch.equal(a, b)


def test_other_planes_take_the_general_path(pkg):
    import torch
    calls = pkg._lib.calls()
    x, f = _planes((8, 6, 4), 1), _planes((8, 6, 4), 2)
    assert calls.rollout_step([t.double() for t in x], f, 1.0) is None
    assert calls.rollout_step([t.transpose(1, 2) for t in x], f, 1.0) is None
    assert calls.rollout_step([t.clone().requires_grad_() for t in x], f, 1.0) is None
    assert calls.rollout_step([t[:7] for t in x], f, 1.0) is None
    with torch.no_grad():
        assert calls.rollout_step([t.clone().requires_grad_() for t in x], f, 1.0) is not None
    inst = pkg.synthetic.land_instance(3, 12, 6, 8)
    st, fo, ge, da = pkg.instance_to_device(inst, "cuda")
    ct = pkg.PhysicsTendency(*_planes((8, 12, 6), 9))
    strided = pkg.PhysicsTendency(*(getattr(ct, k).transpose(1, 2).contiguous().transpose(1, 2)
                                    for k in EVOLVED))
    a = pkg.rollout.rollout_vjp(None, st, fo, ge, da, ct, nsteps=3, checkpoint_every=2)
    b = pkg.rollout.rollout_vjp(None, st, fo, ge, da, strided, nsteps=3, checkpoint_every=2)
    for k in EVOLVED + ("geopotential", "normalized_surface_pressure"):
        assert torch.equal(getattr(a[1], k), getattr(b[1], k)), k
