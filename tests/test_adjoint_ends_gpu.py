"""The device adjoint where a parameter or a field stands at an end of its range: entrainment off
(entmax = 0), a process switched off by an infinite time or scale, equal geopotentials at the two
lowest levels (an infinite gradient of the dry static energy), against the host builds of the
hand-written reverse pass; and its division against IEEE division.

The bar is that of tests/test_adjoint_tiles_gpu.py: each gradient plane within 1e-4 of its largest
value, or three times the host float32 build's own distance from float64; each parameter's sum
within 1e-4 of it, or twice the columns' float32 distances from float64."""
import importlib

import numpy as np
import pytest

from oracle import speedy_oracle as O
from tests.test_adjoint_cpu import (VJP_HAND32, VJP_HAND64, _flags, build_host, column_of,
                                    structs, vjp_any)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pkg():
    return importlib.import_module("jax-gcm_b200")


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    return build_host(tmp_path_factory.mktemp("hostcol") / "libhostcol.so")


def check(pkg, host, inst, **values):
    """GPU VJP of ``inst`` with the parameters ``group__name=value`` against both host builds;
    returns the GPU's parameter gradients."""
    import torch
    kx, ix, il = inst.kx, inst.ix, inst.il
    oracle = {k.replace("__", "."): v for k, v in values.items()}
    tend, data = O.compute_tendencies(*inst.oracle_args(O.default_parameters(**oracle)))
    S = int(sum(1 << int(l) for l in np.nonzero(O.cloud_top_level_set(
        data.shortwave_rad.icltop, kx))[0]))
    vg, _ = structs(pkg, inst)
    parameters = pkg.Parameters.default().with_values(**values)
    pr = parameters.to_struct()
    rng = np.random.default_rng(kx)
    cts = {k: rng.normal(size=(kx, ix, il)).astype(np.float32) for k in "uvtq"}
    state, forcing, geom, date = pkg.instance_to_device(inst, "cuda")
    t = lambda a: torch.as_tensor(a, device="cuda")
    gs, gp = pkg.adjoint.vjp(pkg.SpeedyPhysics(parameters, diagnostics=False), state, forcing,
                             geom, date, pkg.PhysicsTendency(*(t(cts[k]) for k in "uvtq")))
    got = dict(t=gs.temperature, q=gs.specific_humidity, phi=gs.geopotential,
               psa=gs.normalized_surface_pressure, u=gs.u_wind, v=gs.v_wind)
    got = {k: v.cpu().numpy().astype(np.float64) for k, v in got.items()}
    gp = gp.cpu().numpy().astype(np.float64)
    modes = (VJP_HAND64, VJP_HAND32)
    want = {m: {n: np.zeros_like(v) for n, v in got.items()} for m in modes}
    par = {m: np.zeros((ix * il, 12)) for m in modes}
    for i in range(ix):
        for j in range(il):
            h = column_of(inst, data, S, i, j, _flags(inst))
            pad = [0.0] * (16 - kx)
            ct = ([float(x) for x in cts["t"][:, i, j]] + pad,
                  [float(x) for x in cts["q"][:, i, j]] + pad,
                  float(cts["u"][-1, i, j]), float(cts["v"][-1, i, j]))
            for m in modes:
                g = vjp_any(host, m, vg, pr, h, ct)
                par[m][i * il + j] = g["params"]
                for n in ("t", "q", "phi"):
                    want[m][n][:, i, j] = g[n][:kx]
                for n in ("psa", "u", "v"):
                    at = (i, j) if n == "psa" else (-1, i, j)
                    want[m][n][at] = g[n][0]
    w64, w32 = (want[m] for m in modes)
    for n, v in got.items():
        ok = np.isfinite(w64[n])
        assert np.array_equal(np.isfinite(v), ok), (values, n)
        scale = max(np.abs(w64[n][ok]).max(), 1e-30)
        tol = max(1e-4, 3 * np.abs(w32[n][ok] - w64[n][ok]).max() / scale)
        err = np.abs(v[ok] - w64[n][ok]).max() / scale
        assert err <= tol, (values, n, err, tol)
    p64, p32 = (par[m] for m in modes)
    total = p64.sum(0)
    bar = np.maximum(1e-4 * np.abs(total), 2 * np.abs(p32 - p64).sum(0)) + 1e-30
    assert (np.abs(gp - total) <= bar).all(), (values, gp, total, bar)
    return gp


@pytest.mark.parametrize("kx", [7, 8, 16])
def test_no_entrainment(pkg, host, kx):
    inst = pkg.synthetic.land_instance(31 * kx + 43, 43, 3, kx)
    gp = check(pkg, host, inst, convection__entmax=0.0)
    assert gp[4] != 0.0  # the derivative at zero is one-sided and finite


@pytest.mark.parametrize("kx", [7, 8, 16])
@pytest.mark.parametrize("name", ["convection__trcnv", "condensation__trlsc",
                                  "surface_flux__hdrag"])
def test_process_switched_off(pkg, host, kx, name):
    inst = pkg.synthetic.land_instance(31 * kx + 43, 43, 3, kx)
    check(pkg, host, inst, **{name: float("inf")})


@pytest.mark.parametrize("kx", [7, 8, 16])
def test_equal_lowest_geopotentials(pkg, host, kx):
    inst = pkg.synthetic.land_instance(31 * kx + 43, 43, 3, kx)
    inst.phi[-2] = inst.phi[-1]
    check(pkg, host, inst)


def divide(pkg, a, b):
    """The device's a / b, 1 / b and a / b by the full form, and IEEE's a / b and 1 / b."""
    import ctypes as C
    import torch
    on = lambda x: torch.as_tensor(x, dtype=torch.float32, device="cuda")
    x, y, out = on(a), on(b), torch.empty(3, len(a), device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())
    rc = pkg._lib.load().spd_selftest_division(
        len(a), p(x), p(y), p(out), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    with np.errstate(all="ignore"):
        return (*out.cpu().numpy(), a / b, np.float32(1) / b)


def test_division_rounds_like_ieee(pkg):
    """Operands and quotients far from the ends of the exponent range.  The residual of a quotient
    within an ulp is exact, so the corrected one is within half an ulp and a little: never more
    than an ulp from IEEE's, and other than IEEE's only where that little decides (at most one in
    a million is asked for).  The reciprocal has one rounding after its Newton step: one ulp.
    The full form gives the same bits here."""
    rng = np.random.default_rng(20261205)
    n = 1 << 24
    draw = lambda: (rng.uniform(1.0, 2.0, n) * np.exp2(rng.integers(-40, 41, n))
                    * rng.choice([-1.0, 1.0], n)).astype(np.float32)
    short, r, full, q0, r0 = divide(pkg, draw(), draw())
    assert np.array_equal(short.view(np.int32), full.view(np.int32))
    ulps = lambda x, y: np.abs(x.view(np.int32).astype(np.int64) - y.view(np.int32))
    assert ulps(r, r0).max() <= 1
    d = ulps(short, q0)
    assert d.max() <= 1 and (d != 0).sum() <= n // 1000000, (d.max(), (d != 0).sum())


def test_division_at_the_ends(pkg):
    """The full form on every pair of zeros, infinities, NaN and finite values up to 2^125 in size:
    IEEE's result, but for an ulp of a subnormal one; and the two exceptions, a subnormal divisor
    (counts as zero) and one above 2^126 (counts as infinite)."""
    f = np.float32
    size = np.array([0.0, np.inf, np.nan, 1.0, 3.0, 1e-30, 1e30, 2.0 ** -126, 2.0 ** 125], f)
    e = np.concatenate([size, -size])
    a, b = (x.ravel().copy() for x in np.meshgrid(e, e))
    _, _, got, want, _ = divide(pkg, a, b)
    same = (got == want) | (np.isnan(got) & np.isnan(want))
    with np.errstate(invalid="ignore"):
        same |= np.abs(got.astype(float) - want.astype(float)) <= 2.0 ** -149
    assert same.all(), [t for t, s in zip(zip(a, b, got, want), same) if not s]
    x, y = np.array([1.0, 1.0, 1e-39, 2.0 ** 127], f), np.array([1e-39, 2.0 ** 127] * 2, f)
    assert np.array_equal(divide(pkg, x, y)[2], np.array([np.inf, 0.0, np.inf, 0.0], f))
