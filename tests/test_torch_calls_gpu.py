"""What the calls accept as tensors: other dtypes, strides and devices are brought to contiguous
float32 on the state's device and give the same bits as tensors that are that already; results are
contiguous float32 whatever the inputs were; missing or overlapping output tensors are refused."""
import importlib

import pytest

pytestmark = pytest.mark.gpu
STATE = ("u_wind", "v_wind", "temperature", "specific_humidity", "geopotential",
         "normalized_surface_pressure")
TENDENCY = STATE[:4]


@pytest.fixture(scope="module")
def pkg():
    return importlib.import_module("jax-gcm_b200")


@pytest.fixture(scope="module")
def case(pkg):
    inst = pkg.synthetic.land_instance(3, 24, 12, 8)
    return pkg.instance_to_device(inst, "cuda")


def _forms():
    strided = lambda t: t.transpose(-1, -2).contiguous().transpose(-1, -2)
    return {"double": lambda t: t.double(), "strided": strided, "cpu": lambda t: t.cpu(),
            "grad": lambda t: t.clone().requires_grad_(True)}


@pytest.mark.parametrize("form", ["double", "strided", "cpu", "grad"])
def test_inputs_are_brought_to_the_device(pkg, case, form):
    import torch
    st, fo, ge, da = case
    f = _forms()[form]
    keep = (lambda t: t) if form == "cpu" else f  # the state's temperature names the device
    st2 = pkg.PhysicsState(*(keep(getattr(st, n)) if n == "temperature" else f(getattr(st, n))
                             for n in STATE))
    fo2 = pkg.ForcingData(*(f(getattr(fo, n)) for n in (
        "alb0", "sice_am", "snowc_am", "soilw_am", "stl_am", "sea_surface_temperature")),
        lfluxland=fo.lfluxland)
    phys = pkg.SpeedyPhysics()
    want, data = phys.compute_tendencies(st, fo, ge, da)
    got, data2 = phys.compute_tendencies(st2, fo2, ge, da)
    for n in TENDENCY:
        g = getattr(got, n)
        assert g.dtype == torch.float32 and g.is_contiguous() and not g.requires_grad
        assert torch.equal(g, getattr(want, n)), n
    assert data2.convection.iptop.dtype == torch.int32
    assert torch.equal(data2.surface_flux.tskin, data.surface_flux.tskin)
    gen = torch.Generator(device="cuda").manual_seed(1)
    ct = [torch.randn(st.temperature.shape, generator=gen, device="cuda") for _ in range(4)]
    gw, pw = pkg.adjoint.vjp(phys, st, fo, ge, da, pkg.PhysicsTendency(*ct))
    gg, pg = pkg.adjoint.vjp(phys, st2, fo2, ge, da,
                             pkg.PhysicsTendency(*(f(t).detach() for t in ct)))
    for n in STATE:
        g = getattr(gg, n)
        assert g.dtype == torch.float32 and g.is_contiguous() and g.is_cuda
        assert torch.equal(g, getattr(gw, n)), n
    hs = pkg.HeldSuarezPhysics()
    a, b = hs.compute_tendencies(st, geometry=ge)[0], hs.compute_tendencies(st2, geometry=ge)[0]
    for n in TENDENCY:
        assert torch.equal(getattr(a, n), getattr(b, n)), n


def test_output_tensors_are_checked(pkg, case):
    import torch
    st, fo, ge, da = case
    phys = pkg.SpeedyPhysics(diagnostics=False)
    new = lambda n: torch.empty_like(st.temperature if n in TENDENCY else
                                     st.normalized_surface_pressure)
    out = {n: new(n) for n in TENDENCY + ("precnv", "precls")}
    tend, data = phys.compute_tendencies(st, fo, ge, da, out=out)
    assert tend.temperature is out["temperature"] and data.condensation.precls is out["precls"]
    assert data.shortwave_rad.rsds is None
    with pytest.raises(pkg._lib.SpeedyLibraryError):
        phys.compute_tendencies(st, fo, ge, da, out={k: v for k, v in out.items()
                                                      if k != "temperature"})
    with pytest.raises(pkg._lib.SpeedyLibraryError):
        phys.compute_tendencies(st, fo, ge, da, out=dict(out, temperature=st.temperature))
    with pytest.raises(RuntimeError):
        phys.compute_tendencies(pkg.PhysicsState(*(getattr(st, n).cpu() for n in STATE)), fo, ge,
                                da)
