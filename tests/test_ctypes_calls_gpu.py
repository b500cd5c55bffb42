"""The calls through ctypes give the bits of the native ones."""
import importlib

import pytest

pytestmark = pytest.mark.gpu
STATE = ("u_wind", "v_wind", "temperature", "specific_humidity", "geopotential",
         "normalized_surface_pressure")


@pytest.mark.parametrize("kx,ix,il", [(7, 5, 3), (16, 24, 12)])
def test_same_bits(monkeypatch, kx, ix, il):
    import torch
    pkg = importlib.import_module("jax-gcm_b200")
    slow = importlib.import_module("jax-gcm_b200.ctypes_calls")
    case = pkg.instance_to_device(pkg.synthetic.land_instance(3, ix, il, kx), "cuda")
    st, fo, ge, da = case
    ct = pkg.PhysicsTendency(*(torch.randn(kx, ix, il, device="cuda") for _ in range(4)))
    strided = st.copy(temperature=st.temperature.transpose(1, 2).contiguous().transpose(1, 2),
                      geopotential=st.geopotential.double())

    def run():
        got = []
        for diagnostics in (False, True):
            phys = pkg.SpeedyPhysics(diagnostics=diagnostics)
            for s in (st, strided):
                tend, data = phys.compute_tendencies(s, fo, ge, da)
                got += [getattr(tend, n) for n in STATE[:4]]
                got += [data.condensation.precls, data.convection.precnv]
            if diagnostics:
                got += [data.shortwave_rad.rsds, data.surface_flux.tskin, data.convection.iptop]
        out = {k: torch.empty_like(st.temperature) for k in STATE[:4]}
        out.update({k: torch.empty(ix, il, device="cuda") for k in ("precnv", "precls")})
        tend, _ = phys.compute_tendencies(st, fo, ge, da, out=out)
        assert tend.temperature is out["temperature"]
        got += list(out.values())
        for s in (st, strided):
            gs, gp = pkg.adjoint.vjp(phys, s, fo, ge, da, ct)
            got += [getattr(gs, n) for n in STATE]
        got += [getattr(pkg.HeldSuarezPhysics().compute_tendencies(st, geometry=ge)[0], n)
                for n in STATE[:4]]
        final, g, _ = pkg.rollout.rollout_vjp(phys, st, fo, ge, da, ct, nsteps=3,
                                              checkpoint_every=2)
        got += [getattr(final, n) for n in STATE[:4]] + [getattr(g, n) for n in STATE]
        return got

    want = run()
    monkeypatch.setattr(pkg._lib, "_calls", slow)
    got = run()
    assert len(got) == len(want)
    for i, (a, b) in enumerate(zip(got, want)):
        assert a.dtype == b.dtype and torch.equal(a, b), i
