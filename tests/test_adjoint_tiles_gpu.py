"""The adjoint's tiles at the sizes where they can go wrong: one column, less than a warp, one
column past a tile, a last tile of a few columns; gradients written over the cotangents; and the
register budgets, chosen by the batch's warps and levels, bit for bit.

Each column against the host builds of the hand-written reverse pass, with the bar of
tests/test_adjoint_gpu.py: 1e-4 of the field's largest gradient, or three times the host float32
build's own distance from float64 where that is more."""
import ctypes as C
import importlib

import numpy as np
import pytest

from tests.test_adjoint_cpu import (VJP_HAND32, VJP_HAND64, _flags, build_host, column_of,
                                    run_oracle, structs, vjp_any)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pkg():
    return importlib.import_module("jax-gcm_b200")


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    return build_host(tmp_path_factory.mktemp("hostcol") / "libhostcol.so")


@pytest.mark.parametrize("ix,il,kx", [(1, 1, 8), (5, 3, 16), (43, 3, 7), (43, 3, 16), (26, 10, 8)])
def test_ragged_tiles_match_host(pkg, host, ix, il, kx):
    import torch
    inst = pkg.synthetic.land_instance(31 * kx + ix, ix, il, kx)
    tend, data, S = run_oracle(inst)
    vg, pr = structs(pkg, inst)
    rng = np.random.default_rng(ix)
    cts = {k: rng.normal(size=(kx, ix, il)).astype(np.float32) for k in "uvtq"}
    state, forcing, geom, date = pkg.instance_to_device(inst, "cuda")
    phys = pkg.SpeedyPhysics(diagnostics=False)
    t = lambda a: torch.as_tensor(a, device="cuda")
    cot = pkg.PhysicsTendency(t(cts["u"]), t(cts["v"]), t(cts["t"]), t(cts["q"]))
    gs, gp = pkg.adjoint.vjp(phys, state, forcing, geom, date, cot)
    got = dict(t=gs.temperature, q=gs.specific_humidity, phi=gs.geopotential,
               psa=gs.normalized_surface_pressure, u=gs.u_wind, v=gs.v_wind)
    got = {k: v.cpu().numpy().astype(np.float64) for k, v in got.items()}
    want = {k: {n: np.zeros_like(v) for n, v in got.items()} for k in (False, True)}
    par = {False: np.zeros(12), True: np.zeros(12)}
    spread = np.zeros(12)
    for i in range(ix):
        for j in range(il):
            h = column_of(inst, data, S, i, j, _flags(inst))
            ct = ([float(x) for x in cts["t"][:, i, j]] + [0.0] * (16 - kx),
                  [float(x) for x in cts["q"][:, i, j]] + [0.0] * (16 - kx),
                  float(cts["u"][-1, i, j]), float(cts["v"][-1, i, j]))
            one = {}
            for f32, kind in ((False, VJP_HAND64), (True, VJP_HAND32)):
                g = vjp_any(host, kind, vg, pr, h, ct)
                one[f32] = np.array(g["params"])
                par[f32] += one[f32]
                for n in ("t", "q", "phi"):
                    want[f32][n][:, i, j] = g[n][:kx]
                want[f32]["psa"][i, j] = g["psa"][0]
                want[f32]["u"][-1, i, j], want[f32]["v"][-1, i, j] = g["u"][0], g["v"][0]
            spread += np.abs(one[True] - one[False])
    for n, v in got.items():
        scale = max(np.abs(want[False][n]).max(), 1e-30)
        tol = max(1e-4, 3 * np.abs(want[True][n] - want[False][n]).max() / scale)
        err = np.abs(v - want[False][n]).max() / scale
        assert err <= tol, (n, err, tol)
    gp = gp.cpu().numpy().astype(np.float64)
    bar = np.maximum(1e-4 * np.abs(par[False]), 2 * spread) + 1e-30
    assert (np.abs(gp - par[False]) <= bar).all(), (gp, par[False], bar)


def test_gradients_may_overwrite_the_cotangents(pkg):
    """spd_vjp with the gradient planes in the cotangents' own buffers gives the same bits: a
    column reads each level's cotangents before it writes that level."""
    import torch
    L = pkg._lib
    lib = L.load()
    ix, il, kx = 43, 9, 16
    inst = pkg.synthetic.land_instance(5, ix, il, kx)
    state, forcing, geom, date = pkg.instance_to_device(inst, "cuda")
    phys = pkg.SpeedyPhysics(diagnostics=False, fuse_verify=True, time_step=1800.0)
    gen = torch.Generator(device="cuda").manual_seed(2)
    names = ("u_wind", "v_wind", "temperature", "specific_humidity")
    ct = {n: torch.randn(kx, ix, il, generator=gen, device="cuda") for n in names}
    want, want_p = pkg.adjoint.vjp(phys, state, forcing, geom, date, pkg.PhysicsTendency(**ct))
    buf = {n: t.clone() for n, t in ct.items()}
    phi, psa = torch.empty_like(state.geopotential), torch.empty(ix, il, device="cuda")
    par = torch.empty(12, device="cuda")
    owner = lambda n: next(o for o in (state, forcing, geom) if hasattr(o, n))
    inp = L.Inputs(*(getattr(owner(n), n).data_ptr() for n in L.INPUT_FIELDS))
    cts = L.Cotangents(**{n: t.data_ptr() for n, t in buf.items()})
    grads = L.Grads(**{n: t.data_ptr() for n, t in buf.items()}, geopotential=phi.data_ptr(),
                    normalized_surface_pressure=psa.data_ptr(), params=par.data_ptr())
    desc = phys.desc(geom, date, True)
    n = lib.spd_vjp_scratch_bytes(C.byref(desc))
    scratch = torch.empty(n, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    rc = lib.spd_vjp(C.byref(desc), C.byref(geom.vgrid()), C.byref(phys._pstruct), C.byref(inp),
                     C.byref(cts), C.byref(grads), C.c_void_p(scratch.data_ptr()), n,
                     C.c_void_p(stream))
    assert rc == 0
    for f in names:
        assert torch.equal(buf[f], getattr(want, f)), f
    assert torch.equal(phi, want.geopotential)
    assert torch.equal(psa, want.normalized_surface_pressure)


@pytest.mark.parametrize("kx", [7, 8, 16])
def test_register_budgets_give_the_same_bits(pkg, kx):
    """16,384 columns run two warps per scheduler, the 65,536 columns that contain them three or
    four: the same columns' state gradients are equal in every bit."""
    import torch
    il = 256
    inst = pkg.synthetic.land_instance(77, 256, il, kx)
    state, forcing, geom, date = pkg.instance_to_device(inst, "cuda")
    phys = pkg.SpeedyPhysics(diagnostics=False, fuse_verify=True, time_step=1800.0)
    gen = torch.Generator(device="cuda").manual_seed(3)
    ct = [torch.randn(kx, 256, il, generator=gen, device="cuda") for _ in range(4)]
    whole, _ = pkg.adjoint.vjp(phys, state, forcing, geom, date, pkg.PhysicsTendency(*ct))
    cut = lambda t: t[..., :64, :].contiguous()
    names = ("u_wind", "v_wind", "temperature", "specific_humidity", "geopotential",
             "normalized_surface_pressure")
    st = pkg.PhysicsState(*(cut(getattr(state, n)) for n in names))
    fo = pkg.ForcingData(*(cut(getattr(forcing, n)) for n in (
        "alb0", "sice_am", "snowc_am", "soilw_am", "stl_am", "sea_surface_temperature")),
        lfluxland=forcing.lfluxland)
    ge = pkg.Geometry.from_grid_shape((64, il), kx, latitudes=inst.lat, device="cuda")
    ge.orog, ge.phis0, ge.fmask = cut(geom.orog), cut(geom.phis0), cut(geom.fmask)
    ge.sia, ge.coa = geom.sia, geom.coa
    part, _ = pkg.adjoint.vjp(phys, st, fo, ge, date,
                              pkg.PhysicsTendency(*(cut(t) for t in ct)))
    for n in names:
        assert torch.equal(getattr(part, n), cut(getattr(whole, n))), n
