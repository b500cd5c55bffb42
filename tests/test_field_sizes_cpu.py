"""The native calls, and the same through ctypes, refuse a field that holds fewer values than the geometry has, before anything
reaches the library (nothing is launched: every tensor here is on the host, and the last check, for
the device, refuses them too)."""
import ctypes as C
import importlib

import pytest
import torch

pkg = importlib.import_module("jax-gcm_b200")
L = pkg._lib
KX, IX, IL = 8, 6, 4
STATE = ("u_wind", "v_wind", "temperature", "specific_humidity", "geopotential",
         "normalized_surface_pressure")
SURFACE = ("alb0", "sice_am", "snowc_am", "soilw_am", "stl_am", "sea_surface_temperature")
TENDENCY = STATE[:4]


@pytest.fixture(scope="module", params=["native", "ctypes"])
def calls(request):
    if request.param == "native":
        return L.calls()
    return importlib.import_module("jax-gcm_b200.ctypes_calls")


def objects():
    inst = pkg.synthetic.land_instance(3, IX, IL, KX)
    return pkg.instance_to_device(inst, "cpu")


def arguments(phys, ge, da, fo):
    d, vg = phys.desc(ge, da, fo.lfluxland), ge.vgrid()
    return (d, vg), (C.addressof(d), C.addressof(vg), C.addressof(phys._pstruct))


def fwd(calls, st, fo, ge, da, out=None, flags=0):
    phys = pkg.SpeedyPhysics()
    keep, (d, vg, p) = arguments(phys, ge, da, fo)
    keep[0].flags |= flags
    return calls.fwd(st, fo, ge, out, True, d, vg, p, 256, 256, 0)


def vjp(calls, st, fo, ge, da, ct):
    phys = pkg.SpeedyPhysics()
    keep, (d, vg, p) = arguments(phys, ge, da, fo)
    n = L.load().spd_vjp_scratch_bytes(C.byref(keep[0]))
    return calls.vjp(st, fo, ge, ct, d, vg, p, n)


def short(t):
    return t.reshape(-1)[:-1]


def test_host_tensors_of_the_right_size_stop_at_the_device(calls):
    st, fo, ge, da = objects()
    ct = pkg.PhysicsTendency(*(torch.zeros(KX, IX, IL) for _ in range(4)))
    with pytest.raises(RuntimeError, match="CUDA"):
        fwd(calls, st, fo, ge, da)
    with pytest.raises(RuntimeError, match="CUDA"):
        vjp(calls, st, fo, ge, da, ct)
    hs = pkg.HeldSuarezPhysics()
    d = hs._desc(ge)
    with pytest.raises(RuntimeError, match="CUDA"):
        calls.held_suarez(st, hs._lat_table(ge, "cpu"), None, C.addressof(d))


@pytest.mark.parametrize("name", STATE + SURFACE + ("fmask", "orog", "phis0", "sia", "coa"))
def test_short_inputs(calls, name):
    st, fo, ge, da = objects()
    owner = next(o for o in (st, fo, ge) if hasattr(o, name))
    setattr(owner, name, short(getattr(owner, name)))
    ct = pkg.PhysicsTendency(*(torch.zeros(KX, IX, IL) for _ in range(4)))
    for call in (lambda: fwd(calls, st, fo, ge, da), lambda: vjp(calls, st, fo, ge, da, ct)):
        with pytest.raises(ValueError, match=name):
            call()


def test_lowest_level_winds_need_one_level(calls):
    st, fo, ge, da = objects()
    st.u_wind, st.v_wind = st.u_wind[-1], st.v_wind[-1]
    with pytest.raises(RuntimeError, match="CUDA"):
        fwd(calls, st, fo, ge, da, flags=L.SPD_LOW_LEVEL_WINDS)
    st.v_wind = short(st.v_wind)
    with pytest.raises(ValueError, match="v_wind"):
        fwd(calls, st, fo, ge, da, flags=L.SPD_LOW_LEVEL_WINDS)


@pytest.mark.parametrize("name", TENDENCY)
def test_short_cotangents(calls, name):
    st, fo, ge, da = objects()
    ct = pkg.PhysicsTendency(*(torch.zeros(KX, IX, IL) for _ in range(4)))
    setattr(ct, name, short(getattr(ct, name)))
    with pytest.raises(ValueError, match=name):
        vjp(calls, st, fo, ge, da, ct)


@pytest.mark.parametrize("field", L.OUTPUT_FIELDS)
def test_short_outputs(calls, field):
    st, fo, ge, da = objects()
    out = [torch.zeros((KX, IX, IL) if f in TENDENCY else (IX, IL),
                       dtype=torch.int32 if f in ("iptop", "icltop") else torch.float32)
           for f in L.OUTPUT_FIELDS]
    with pytest.raises(RuntimeError, match="CUDA"):
        fwd(calls, st, fo, ge, da, out)
    i = L.OUTPUT_FIELDS.index(field)
    # a view that ends before the plane does, and one whose elements lie on one another
    for bad in (short(out[i]).clone(), torch.zeros(1, dtype=out[i].dtype).expand(out[i].shape)):
        with pytest.raises(ValueError, match=field):
            fwd(calls, st, fo, ge, da, out[:i] + [bad] + out[i + 1:])


@pytest.mark.parametrize("name", ("u_wind", "v_wind", "temperature",
                                  "normalized_surface_pressure", "out", "table"))
def test_held_suarez(calls, name):
    st, fo, ge, da = objects()
    hs = pkg.HeldSuarezPhysics()
    d, tab, out = hs._desc(ge), hs._lat_table(ge, "cpu"), None
    if name == "out":
        out = [torch.zeros(KX, IX, IL) for _ in range(3)] + [torch.zeros(KX, IX, IL - 1)]
    elif name == "table":
        tab = tab[:, :-1].contiguous()
    else:
        setattr(st, name, short(getattr(st, name)))
    with pytest.raises(ValueError):
        calls.held_suarez(st, tab, out, C.addressof(d))


@pytest.mark.parametrize("name", STATE + SURFACE + ("fmask", "orog", "phis0", "sia", "coa"))
def test_short_ensemble_inputs(monkeypatch, name):
    monkeypatch.setattr(L, "preload", lambda index: None)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    st, fo, ge, da = objects()
    owner = next(o for o in (st, fo, ge) if hasattr(o, name))
    setattr(owner, name, short(getattr(owner, name)))
    with pytest.raises(ValueError, match=name):
        pkg.Ensemble([pkg.Member(st, fo, ge)], da)


@pytest.mark.parametrize("name", TENDENCY + ("precnv", "rsds", "icltop"))
def test_short_ensemble_outputs(monkeypatch, name):
    monkeypatch.setattr(L, "preload", lambda index: None)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    st, fo, ge, da = objects()
    out = {f: torch.zeros((KX, IX, IL) if f in TENDENCY else (IX, IL)) for f in L.OUTPUT_FIELDS}
    out[name] = short(out[name]).clone()
    with pytest.raises(ValueError, match=name):
        pkg.Ensemble([pkg.Member(st, fo, ge, out)], da)
