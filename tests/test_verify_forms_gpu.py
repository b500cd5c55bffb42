"""The fused launch's forms (two or four blocks per SM, with and without verify): the call with
verify fused against the call without it on the clamped state, limited afterwards.

Everything but a limited level's humidity tendency, -q / dt, is the same arithmetic and equal in
every bit; the kernel divides with the hardware's division (2 ulp), so those agree to 3e-7."""
import importlib

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kx,ix,il", [(7, 43, 3), (8, 1, 1), (16, 95, 47), (7, 300, 256),
                                      (8, 300, 256), (16, 300, 257)])
@pytest.mark.parametrize("share", [0.0, 0.3, 1.0])
def test_verify_equals_limiting_afterwards(kx, ix, il, share):
    import torch
    pkg = importlib.import_module("jax-gcm_b200")
    inst = pkg.synthetic.land_instance(11 + kx, ix, il, kx)
    st, fo, ge, da = pkg.instance_to_device(inst, "cuda")
    gen = torch.Generator(device="cuda").manual_seed(kx)
    q = st.specific_humidity
    q = torch.where(torch.rand(q.shape, generator=gen, device="cuda") < share, -0.3 * q - 1e-3, q)
    dt = 1800.0
    got, data = pkg.SpeedyPhysics(fuse_verify=True, time_step=dt).compute_tendencies(
        st.copy(specific_humidity=q), fo, ge, da)
    clamped = torch.where(q < 0, torch.zeros_like(q), q)
    want, data2 = pkg.SpeedyPhysics().compute_tendencies(st.copy(specific_humidity=clamped), fo,
                                                         ge, da)
    for n in ("u_wind", "v_wind", "temperature"):
        assert torch.equal(getattr(got, n), getattr(want, n)), n
    for a, b in ((data.surface_flux.tskin, data2.surface_flux.tskin),
                 (data.condensation.precls, data2.condensation.precls)):
        assert torch.equal(a, b)
    dq = want.specific_humidity
    keep = q + dt * dq >= 0
    assert torch.equal(got.specific_humidity[keep], dq[keep])
    lim = -q[~keep] / dt
    assert ((got.specific_humidity[~keep] - lim).abs() <= 3e-7 * lim.abs()).all()
