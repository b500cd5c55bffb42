"""The structures whose addresses the native calls get live until the call returns, also where the
geometry makes a new one for each call or the physics' parameters are replaced meanwhile."""
import importlib
import weakref
from types import SimpleNamespace

import pytest
import torch

pkg = importlib.import_module("jax-gcm_b200")
L = pkg._lib
physics = importlib.import_module("jax-gcm_b200.physics")
adjoint = importlib.import_module("jax-gcm_b200.adjoint")


class FreshGeometry:
    def __init__(self, geometry, made):
        self.geometry, self.made = geometry, made

    def __getattr__(self, name):
        return getattr(self.geometry, name)

    def vgrid(self):
        vg = L.VGrid()
        self.made.append(weakref.ref(vg))
        return vg


@pytest.mark.parametrize("kind", ["forward", "adjoint"])
def test_structures_outlive_the_call(monkeypatch, kind):
    inst = pkg.synthetic.land_instance(3, 4, 2, 8)
    st, fo, ge, da = pkg.instance_to_device(inst, "cpu")
    phys, made = pkg.SpeedyPhysics(), []
    made.append(weakref.ref(phys._pstruct))

    def call(*args):
        phys._pstruct = L.Params()  # another thread sets new parameters
        assert len(made) == 2 and all(r() is not None for r in made)
        return 0, [None] * 21

    monkeypatch.setattr(L, "calls", lambda: SimpleNamespace(fwd=call, vjp=call))
    monkeypatch.setattr(L, "preload", lambda index: None)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(physics, "current_raw_stream", lambda index: 0)
    st.temperature = SimpleNamespace(shape=st.temperature.shape, is_cuda=True,
                                     device=torch.device("cpu"), get_device=lambda: 0)
    geom = FreshGeometry(ge, made)
    if kind == "forward":
        phys.compute_tendencies(st, fo, geom, da)
    else:
        adjoint.vjp(phys, st, fo, geom, da, None)
    assert len(made) == 2
