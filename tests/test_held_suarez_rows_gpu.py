"""The Held-Suarez path for shapes and pointers that 128-bit accesses do not fit: the edges of its
128-column items and of its level pairs against the oracle (the bar of tests/test_held_suarez.py:
1e-5 of the field's largest value), and planes one float off their alignment bit for bit like the
aligned ones."""
import importlib

import numpy as np
import pytest

from oracle import held_suarez_oracle as H

pytestmark = pytest.mark.gpu
NAMES = ("u_wind", "v_wind", "temperature", "specific_humidity")


@pytest.fixture(scope="module")
def pkg():
    return importlib.import_module("jax-gcm_b200")


@pytest.mark.parametrize("kx,ix,il", [(8, 1, 1), (16, 3, 11), (7, 127, 1), (7, 43, 3),
                                      (8, 361, 1), (16, 95, 47)])
def test_ragged_shapes_match_oracle(pkg, kx, ix, il):
    import torch
    inst = pkg.synthetic.land_instance(70 + ix, ix, il, kx)
    st, fo, ge, da = pkg.instance_to_device(inst, "cuda")
    out = {n: torch.full((kx, ix, il), float("nan"), device="cuda") for n in NAMES}
    tend, _ = pkg.HeldSuarezPhysics().compute_tendencies(st, fo, ge, da, out=out)
    ref = H.compute_tendencies(inst.u, inst.v, inst.t, inst.psa, ge.fsg, inst.lat)
    for n, r in zip(NAMES, ref):
        g = getattr(tend, n).cpu().numpy()
        assert np.abs(g - r).max() <= 1e-5 * max(np.abs(r).max(), 1e-30), n


@pytest.mark.parametrize("kx", [7, 16])
def test_misaligned_planes_give_the_same_bits(pkg, kx):
    import torch
    inst = pkg.synthetic.land_instance(5, 64, 32, kx)
    st, fo, ge, da = pkg.instance_to_device(inst, "cuda")
    phys = pkg.HeldSuarezPhysics()
    want, _ = phys.compute_tendencies(st, fo, ge, da)
    off = lambda t: torch.empty(t.numel() + 1, device="cuda")[1:].view(t.shape).copy_(t)
    moved = pkg.PhysicsState(off(st.u_wind), off(st.v_wind), off(st.temperature),
                             st.specific_humidity, st.geopotential,
                             off(st.normalized_surface_pressure))
    assert moved.u_wind.data_ptr() % 16 == 4
    out = {k: off(torch.full((kx, 64, 32), float("nan"), device="cuda")) for k in NAMES}
    got, _ = phys.compute_tendencies(moved, fo, ge, da, out=out)
    for k in NAMES:
        assert torch.equal(getattr(got, k), getattr(want, k)), k
