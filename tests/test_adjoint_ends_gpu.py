"""The device adjoint where a parameter stands at an end of its range: entrainment off
(entmax = 0), against the host builds of the hand-written reverse pass.

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
        scale = max(np.abs(w64[n]).max(), 1e-30)
        tol = max(1e-4, 3 * np.abs(w32[n] - w64[n]).max() / scale)
        err = np.abs(v - w64[n]).max() / scale
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
