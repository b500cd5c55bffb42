"""What a user of the framework has it do, as cases that can be timed and checked.

Physics calls on one grid (``SpeedyPhysics.compute_tendencies``), one fused step of a ragged
ensemble (``Ensemble.forward``), the adjoint (``adjoint.vjp``), a checkpointed rollout gradient
(``rollout.rollout_vjp``) and the Held-Suarez forcing (``HeldSuarezPhysics.compute_tendencies``),
from grids of a few thousand columns, where latency and launches count, to T425 with 16 levels
(819,200 columns).  Inputs are seeded synthetic columns with the value distributions of the
package's own generators, made on the device; ``exact`` evaluates the same physics in float64
with plain torch (and its autograd for the gradients).
"""
from __future__ import annotations

import functools
import importlib
import math

import numpy as np
import torch

spd = importlib.import_module("jax-gcm_b200")

DAYS_YEAR = 365.2425
GRAV, CP, RGAS, ALHC, P0 = 9.81, 1004.0, 2.0 / 7.0 * 1004.0, 2501.0, 1e5
SBC = 5.67e-8

SIGMA = {
    7: [0.0, 0.14, 0.26, 0.42, 0.6, 0.77, 0.9, 1.0],
    8: [0.0, 0.05, 0.14, 0.26, 0.42, 0.6, 0.77, 0.9, 1.0],
    16: [k / 16.0 for k in range(17)],
}
GRIDS = {21: (64, 32), 31: (96, 48), 42: (128, 64), 85: (256, 128), 170: (512, 256),
         425: (1280, 640)}
# (truncation, member count) of the ragged ensemble: 61 members, 466,944 columns
LAYOUT = ((21, 32), (31, 16), (42, 8), (85, 4), (170, 1))


def listed():
    return [
        # the smallest call a model makes: a T21 step's physics, with its diagnostics
        dict(name="call_t21_8", kind="call", ix=64, il=32, kx=8, land=True, verify=False,
             diag=True),
        # a regional or lat-lon grid whose sizes divide nothing, 7 levels, verify fused
        dict(name="call_95x47_7", kind="call", ix=95, il=47, kx=7, land=True, verify=True,
             diag=True),
        # an ordinary model step: T85 with 16 levels, verify fused, tendencies only
        dict(name="call_t85_16", kind="call", ix=256, il=128, kx=16, land=True, verify=True,
             diag=False),
        # the largest call: T425 with 16 levels
        dict(name="call_t425_16", kind="call", ix=1280, il=640, kx=16, land=True, verify=False,
             diag=False),
        # a forecast ensemble of mixed resolutions and level counts, one fused step
        dict(name="ensemble_61", kind="ensemble", scale=1),
        # gradients: parameter estimation at T42, data assimilation at T85 and T170, and the
        # largest grid; T170 with verify fused, as inside a model step
        dict(name="vjp_t42_8", kind="vjp", ix=128, il=64, kx=8, land=True, verify=False),
        dict(name="vjp_t85_16", kind="vjp", ix=256, il=128, kx=16, land=True, verify=False),
        dict(name="vjp_t170_16", kind="vjp", ix=512, il=256, kx=16, land=True, verify=True),
        dict(name="vjp_t425_16", kind="vjp", ix=1280, il=640, kx=16, land=True, verify=False),
        # a training step: the gradient of a 12-step rollout, checkpoints every 4 steps
        dict(name="rollout_t42_8", kind="rollout", ix=128, il=64, kx=8, land=True, nsteps=12,
             every=4),
        # Held-Suarez runs: the largest grid, and a 1-degree grid with both poles and the
        # repeated meridian, whose planes are not a multiple of 16 bytes
        dict(name="hs_t425_16", kind="hs", ix=1280, il=640, kx=16),
        dict(name="hs_361x181_16", kind="hs", ix=361, il=181, kx=16),
    ]


def draw(rng):
    """Another case of the same ranges: grids from 64x32 to 1280x640, odd sizes among them."""
    def size(hi):
        il = int(round(32 * math.exp(rng.random() * math.log(hi / 32.0))))
        ix = int(round(2 * il * rng.uniform(0.95, 1.0)))
        return dict(ix=min(ix, 1280), il=il)

    kind = rng.choice(["call", "call", "call", "vjp", "vjp", "vjp", "hs", "ensemble", "rollout"])
    kx = rng.choice([7, 8, 8, 16, 16])
    land = rng.random() < 0.8
    if kind == "call":
        return dict(kind=kind, **size(640), kx=kx, land=land, verify=rng.random() < 0.5,
                    diag=rng.random() < 0.5)
    if kind == "vjp":
        return dict(kind=kind, **size(640), kx=kx, land=land, verify=rng.random() < 0.5)
    if kind == "hs":
        return dict(kind=kind, **size(640), kx=kx)
    if kind == "rollout":
        return dict(kind=kind, **size(80), kx=kx, land=land, nsteps=rng.choice([6, 9, 12]),
                    every=rng.choice([3, 4]))
    return dict(kind=kind, scale=rng.choice([2, 3, 4, 8]))


# ---------------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=64)
def _latitudes(il):
    x, _ = np.polynomial.legendre.leggauss(il)
    return np.arcsin(x)


@functools.lru_cache(maxsize=None)
def _vertical(kx):
    """Vertical sigma tables, float32 (they are inputs of the physics)."""
    f = np.float32
    hsg = np.asarray(SIGMA[kx], f)
    fsg = (hsg[1:] + hsg[:-1]) / f(2.0)
    dhs = np.diff(hsg)
    sigl = np.log(fsg)
    grdsig = f(GRAV) / (dhs * f(P0))
    grdscp = grdsig / f(CP)
    wvi = np.zeros(kx, f)
    w0 = f(1.0) / np.diff(sigl)
    wvi[:-1] = (np.log(hsg[1:-1]) - sigl[:-1]) * w0
    wvi[-1] = (np.log(f(0.99)) - sigl[-1]) * w0[-1]
    return dict(hsg=hsg, fsg=fsg, dhs=dhs, sigl=sigl, grdsig=grdsig, grdscp=grdscp, wvi=wvi)


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _fields(seed, ix, il, kx, land=True, ringing=False):
    """Fields of one grid, float32 on the device: a lapse-rate atmosphere with noise, humidity
    of 30 to 95 % falling off with height, 30 % land with orography, soil moisture, snow
    poleward of 50 degrees, sea ice where the sea is below 271.4 K; all ocean without land.
    ringing: 2 % of the humidities slightly negative, as a spectral model hands them to the
    physics that clamps them (verify)."""
    dev = _device()
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    f32 = torch.float32
    normal = lambda *s: torch.randn(*s, generator=gen, device=dev, dtype=f32)
    uniform = lambda *s: torch.rand(*s, generator=gen, device=dev, dtype=f32)
    lat = torch.as_tensor(_latitudes(il), dtype=f32, device=dev)
    cos2 = torch.cos(lat) ** 2
    sig = torch.as_tensor(_vertical(kx)["fsg"], device=dev)[:, None, None]
    if land:
        coarse = normal(1, 1, max(4, ix // 12), max(4, il // 12))
        noise = torch.nn.functional.interpolate(coarse, size=(ix, il), mode="bilinear",
                                                align_corners=True)[0, 0]
        cut = noise.reshape(-1).kthvalue(max(1, int(0.7 * ix * il))).values
        fmask = (noise >= cut).to(f32)
    else:
        fmask = torch.zeros(ix, il, device=dev)
    phis = normal(ix, il).abs() * 1.5e4 * fmask
    t = torch.clamp(288.0 + 45.5 * torch.log(sig) + 2.0 * normal(kx, ix, il), min=200.0)
    psa = torch.exp(0.01 * normal(ix, il))
    warm = t >= 273.16
    e = 6.108e-3 * torch.exp(torch.where(warm, 17.269 * (t - 273.16) / (t - 35.86),
                                         21.875 * (t - 273.16) / (t - 7.66)))
    q = (0.3 + 0.65 * uniform(kx, ix, il)) * sig ** 2 * (622.0 * e / (sig * psa - 0.378 * e))
    if ringing:
        q = torch.where(uniform(kx, ix, il) < 0.02, -0.05 * q, q)
    sst = (271.4 + 29.0 * cos2)[None, :].expand(ix, il).contiguous()
    snowy = (lat.abs() > math.radians(50.0)).to(f32)[None, :]
    return dict(
        u=25.0 * cos2 * (1.0 - sig) + 3.0 * normal(kx, ix, il), v=3.0 * normal(kx, ix, il),
        t=t, q=q, phi=phis + RGAS * t * (-torch.log(sig)), psa=psa, sst=sst, stl=sst.clone(),
        soilw=uniform(ix, il) * float(land), snowc=uniform(ix, il) / 0.6 * snowy * fmask,
        sice=(sst < 271.4).to(f32) * float(land),
        alb0=torch.full((ix, il), 0.2 if land else 0.0, device=dev), fmask=fmask,
        orog=phis / GRAV, phis0=phis, sia=torch.sin(lat), coa=torch.cos(lat))


def _cotangent(seed, kx, ix, il):
    gen = torch.Generator(device=_device()).manual_seed(int(seed) + 7919)
    return {k: torch.randn(kx, ix, il, generator=gen, device=_device()) for k in "uvtq"}


def _objects(f, kx, ix, il, land):
    st = spd.PhysicsState(f["u"], f["v"], f["t"], f["q"], f["phi"], f["psa"])
    fo = spd.ForcingData(f["alb0"], f["sice"], f["snowc"], f["soilw"], f["stl"], f["sst"],
                         lfluxland=land)
    ge = spd.Geometry.from_grid_shape((ix, il), kx, latitudes=_latitudes(il), device=_device())
    ge.orog, ge.phis0, ge.fmask = f["orog"], f["phis0"], f["fmask"]
    ge.sia, ge.coa = f["sia"], f["coa"]
    return st, fo, ge


def _date():
    return spd.DateData(tyear=80.0 / DAYS_YEAR, model_year=1950, model_step=0, dt_seconds=1800.0)


def _members(scale):
    """(ix, il, kx) of the ragged ensemble's members, levels alternating 8 and 16 (T170: 16)."""
    out = []
    for trunc, count in LAYOUT:
        for n in range(max(1, count // scale)):
            out.append(GRIDS[trunc] + (16 if trunc == 170 or n % 2 == 1 else 8,))
    return out


ENS_FIELDS = ("u_wind", "v_wind", "temperature", "specific_humidity", "precnv", "precls")


def _ensemble_offsets(members):
    """Offset of every member in the ensemble's flat result buffers (64-float steps) and their
    length, for the level fields and for the surface fields."""
    at, n3, n2 = [], 0, 0
    for ix, il, kx in members:
        at.append((n3, n2))
        n3 += -(-kx * ix * il // 64) * 64
        n2 += -(-ix * il // 64) * 64
    return at, n3, n2


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        members = _members(case["scale"])
        at, n3, n2 = _ensemble_offsets(members)
        flat = {k: torch.zeros(n2 if k in ("precnv", "precls") else n3, device=_device())
                for k in ENS_FIELDS}
        ms = []
        for i, ((ix, il, kx), (o3, o2)) in enumerate(zip(members, at)):
            f = _fields(seed * 1000 + i, ix, il, kx)
            n = ix * il
            out = {k: flat[k][o2:o2 + n].view(ix, il) if k in ("precnv", "precls")
                   else flat[k][o3:o3 + kx * n].view(kx, ix, il) for k in ENS_FIELDS}
            ms.append(spd.Member(*_objects(f, kx, ix, il, True), out))
        return dict(kind=kind, ens=spd.Ensemble(ms, _date()), flat=flat)
    kx, ix, il = case["kx"], case["ix"], case["il"]
    land = case.get("land", True)
    st, fo, ge = _objects(_fields(seed, ix, il, kx, land, case.get("verify", False)), kx, ix, il,
                          land)
    s = dict(kind=kind, state=st, forcing=fo, geometry=ge, date=_date())
    if kind == "hs":
        s["phys"] = spd.HeldSuarezPhysics()
        return s
    s["phys"] = spd.SpeedyPhysics(fuse_verify=case.get("verify", False),
                                  diagnostics=case.get("diag", False))
    if kind in ("vjp", "rollout"):
        ct = _cotangent(seed, kx, ix, il)
        s["ct"] = spd.PhysicsTendency(ct["u"], ct["v"], ct["t"], ct["q"])
    if kind == "rollout":
        s["nsteps"], s["every"] = case["nsteps"], case["every"]
    return s


def _state_dict(x):
    return dict(u=x.u_wind, v=x.v_wind, t=x.temperature, q=x.specific_humidity,
                phi=x.geopotential, psa=x.normalized_surface_pressure)


def run(s):
    kind = s["kind"]
    if kind == "ensemble":
        s["ens"].forward()
        return s["flat"]
    if kind == "hs":
        tend, _ = s["phys"].compute_tendencies(s["state"], geometry=s["geometry"])
        return dict(u=tend.u_wind, v=tend.v_wind, t=tend.temperature, q=tend.specific_humidity)
    if kind == "vjp":
        g, p = spd.adjoint.vjp(s["phys"], s["state"], s["forcing"], s["geometry"], s["date"],
                               s["ct"])
        return dict(_state_dict(g), params=p)
    if kind == "rollout":
        x, g, p = spd.rollout.rollout_vjp(s["phys"], s["state"], s["forcing"], s["geometry"],
                                          s["date"], s["ct"], nsteps=s["nsteps"],
                                          checkpoint_every=s["every"])
        return dict(final=dict(u=x.u_wind, v=x.v_wind, t=x.temperature, q=x.specific_humidity),
                    grad=_state_dict(g), params=p)
    tend, data = s["phys"].compute_tendencies(s["state"], s["forcing"], s["geometry"], s["date"])
    out = dict(u=tend.u_wind, v=tend.v_wind, t=tend.temperature, q=tend.specific_humidity,
               precnv=data.convection.precnv, precls=data.condensation.precls)
    if s["phys"].diagnostics:
        sw, sf = data.shortwave_rad, data.surface_flux
        out.update(iptop=data.convection.iptop, cbmf=data.convection.cbmf, cloudc=sw.cloudc,
                   cloudstr=sw.cloudstr, icltop=sw.icltop, rsds=sw.rsds, rsns=sw.rsns,
                   ftop_sw=sw.ftop, ftop_lw=data.longwave_rad.ftop, rlds=sf.rlds, rlns=sf.rlns,
                   tsfc=sf.tsfc, tskin=sf.tskin, shf=sf.shf, evap=sf.evap)
    return out


def work(case):
    """Bytes: each field the physics reads once (winds at the lowest level only), each output
    once.  Operations: element operations of the column physics (about 245 per level and 240
    per column, an exponential counted as one), three times that for a gradient."""
    kind = case["kind"]
    if kind == "ensemble":
        members = [dict(kind="call", ix=a, il=b, kx=k) for a, b, k in _members(case["scale"])]
        parts = [work(m) for m in members]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    kx, n = case["kx"], case["ix"] * case["il"]
    ops = n * (245 * kx + 240)
    call = 4 * n * (7 * kx + 14 + (15 if case.get("diag") else 0))
    vjp = 4 * n * (10 * kx + 15)
    if kind == "call":
        return dict(bytes=call, flops=ops)
    if kind == "hs":
        return dict(bytes=4 * n * (7 * kx + 1), flops=30 * kx * n)
    if kind == "vjp":
        return dict(bytes=vjp, flops=3 * ops)
    steps = case["nsteps"]
    forwards = 2 * steps - -(-steps // case["every"])
    return dict(bytes=steps * vjp + forwards * call, flops=(3 * steps + forwards) * ops)


# ---------------------------------------------------------------------------------------------
# The physics in float64 (plain torch), columns along the last axis
# ---------------------------------------------------------------------------------------------
_P = dict(psmin=0.8, trcnv=6.0, rhil=0.7, rhbl=0.9, entmax=0.5, smf=0.8, trlsc=4.0, rhlsc=0.9,
          drhlsc=0.1, rhblsc=0.95, albcl=0.43, albcls=0.50)
_R = dict(absdry=0.033, absaer=0.033, abswv1=0.022, abswv2=15.0, abscl1=0.015, abscl2=0.15,
          ablwin=0.3, ablco2=6.0, ablwv1=0.7, ablwv2=50.0, ablcl1=12.0, ablcl2=0.6, rhcl1=0.30,
          rhcl2=1.0, qacl=0.20, wpcl=0.2, pmaxcl=10.0, clsmax=0.60, clsminl=0.15, gse_s0=0.25,
          gse_s1=0.40, albsea=0.07, albice=0.60, albsn=0.60, epslw=0.05, emisfc=0.98, fwind0=0.95,
          ftemp0=1.0, cdl=2.4e-3, cds=1.0e-3, chl=1.2e-3, chs=0.9e-3, vgust=5.0, ctday=1.0e-2,
          dtheta=3.0, fstab=0.67, clambda=7.0, clambsn=7.0, hdrag=2000.0, trshc=6.0, trvdi=24.0,
          trvds=6.0, redshc=0.5, rhgrad=0.5, segrad=0.1)
PARAMS = tuple(_P)
CHUNK = 1 << 16  # columns evaluated at once


def _single(x):
    return float(np.float32(x))


def _qsat(t, ps, sig):
    warm = t >= 273.16
    e = 6.108e-3 * torch.exp(torch.where(warm, 17.269 * (t - 273.16) / (t - 35.86),
                                         21.875 * (t - 273.16) / (t - 7.66)))
    return 622.0 * e / (sig * ps - 0.378 * e)


def _at_least(x, lo):
    return torch.maximum(x, torch.full_like(x, lo))


def _at_most(x, hi):
    return torch.minimum(x, torch.full_like(x, hi))


def _solar(tyear, sia, coa):
    """Daily mean insolation and what goes with it, per column."""
    alpha = 2.0 * math.pi * tyear
    c1, s1 = math.cos(alpha), math.sin(alpha)
    c2, s2 = c1 * c1 - s1 * s1, 2.0 * s1 * c1
    c3, s3 = c1 * c2 - s1 * s2, s1 * c2 + s2 * c1
    decl = (0.006918 - 0.399912 * c1 + 0.070257 * s1 - 0.006758 * c2 + 0.000907 * s2
            - 0.002697 * c3 + 0.001480 * s3)
    fdis = 1.000110 + 0.034221 * c1 + 0.001280 * s1 + 0.000719 * c2 + 0.000077 * s2
    h0 = torch.acos(torch.clamp(-math.tan(decl) * sia / coa, -1.0, 1.0))
    fsol = 1368.0 / math.pi * fdis * (h0 * sia * math.sin(decl)
                                      + torch.sin(h0) * coa * math.cos(decl))
    a2 = 2.0 * math.pi * (tyear + 10.0 / 365.0)
    rzen = -math.cos(a2) * 23.45 * math.pi / 180.0
    flat2 = 1.5 * sia * sia - 0.5
    ozone = 0.4 * 0.02 * (1.0 + max(0.0, math.cos(a2)) * sia + 1.8 * flat2)
    zenit = 1.0 + (1.0 - (coa * math.cos(rzen) + sia * math.sin(rzen))) ** 2
    return dict(fsol=fsol, ozupp=fsol * 0.01 * zenit, ozone=fsol * ozone * zenit, zenit=zenit,
                stratz=torch.clamp(6.0 - fsol, min=0.0))


def _physics(x, b, par, kx, land, verify, dt_seconds, step, levels):
    """Tendencies and diagnostics of columns.  x: state (u, v at the lowest level; t, q, phi as
    lists of levels; psa), b: boundary fields, par: the 12 tuned parameters; levels: the cloud
    reflection levels of the whole grid, or None to return every column's cloud top only."""
    V = {k: [float(a) for a in v] for k, v in _vertical(kx).items()}
    R = {k: _single(v) for k, v in _R.items()}
    hsg, fsg, dhs, wvi = V["hsg"], V["fsg"], V["dhs"], V["wvi"]
    T, PHI, psa = x["t"], x["phi"], x["psa"]
    Qraw = x["q"]
    zero = torch.zeros_like(psa)
    Q = [torch.where(q < 0.0, zero, q) for q in Qraw] if verify else Qraw
    QS = [_qsat(T[k], psa, fsg[k]) for k in range(kx)]
    RH = [Q[k] / QS[k] for k in range(kx)]
    SE = [CP * T[k] + PHI[k] for k in range(kx)]
    DT, DQ = [zero] * kx, [zero] * kx
    B = kx - 1
    # convection: diagnosis
    mse0 = SE[B] + ALHC * Q[B]
    mse1 = torch.minimum(mse0, SE[B - 1] + ALHC * Q[B - 1])
    mss0 = torch.maximum(mse0, SE[B] + ALHC * QS[B])
    ktop1 = torch.full_like(psa, kx, dtype=torch.int64)
    ktop2, msthr = ktop1.clone(), zero
    for k in range(kx - 4, 1, -1):
        m0, m1 = SE[k] + ALHC * QS[k], SE[k + 1] + ALHC * QS[k + 1]
        m = m0 + wvi[k] * (m1 - m0)
        ktop1 = torch.where(mss0 > m, k + 1, ktop1)
        ktop2 = torch.where(mse1 > m, k + 1, ktop2)
        msthr = torch.where(mse1 > m, m, msthr)
    thr0, thr1 = par["rhbl"] * QS[B], par["rhbl"] * QS[B - 1]
    deep = (psa > par["psmin"]) & (ktop1 < kx)
    case1 = deep & (ktop2 < kx)
    case2 = deep & ~(ktop2 < kx) & (Q[B] > thr0) & (Q[B - 1] > thr1)
    qdif = torch.where(case1, torch.maximum(Q[B] - thr0, (mse0 - msthr) / ALHC),
                       torch.where(case2, Q[B] - thr0, zero))
    iptop = torch.where(case1 | case2, ktop1, kx + 1)
    # convection: tendencies
    ent = [max(0.0, fsg[k] - 0.5) ** 2 for k in range(kx)]
    scale = par["entmax"] / sum(ent[1:-1])
    qmax = torch.maximum(1.01 * Q[B], QS[B])
    sb = SE[B - 1] + wvi[B - 1] * (SE[B] - SE[B - 1])
    qb = torch.minimum(Q[B - 1] + wvi[B - 1] * (Q[B] - Q[B - 1]), Q[B])
    fpsa = psa * _at_most((psa - par["psmin"]) * (2.0 / (1.0 - par["psmin"])), 1.0)
    fmass = (P0 * dhs[B] / (GRAV * 3600.0 * par["trcnv"]) * fpsa
             * _at_most(qdif / (qmax - qb), 5.0))
    conv = iptop < kx
    cbmf = torch.where(conv, fmass, zero)
    cm, cs, cq = zero, zero, zero
    fm, fus, fuq, fds, fdq = ([None] * kx for _ in range(5))
    for k in range(B, -1, -1):
        on = (k >= iptop) if k < B else torch.zeros_like(conv)
        en = torch.where(on, ent[k] * scale * psa * cbmf, zero) if 1 <= k < B else zero
        cm, cs, cq = cm + en, cs + en * SE[k], cq + en * Q[k]
        fm[k], fus[k], fuq[k] = fmass + cm, fmass * SE[B] + cs, fmass * qmax + cq
        if k == B:
            fds[k], fdq[k] = fmass * sb, fmass * qb
        elif k > 0:
            fds[k] = fm[k] * (SE[k - 1] + wvi[k - 1] * (SE[k] - SE[k - 1]))
            fdq[k] = fm[k] * (Q[k - 1] + wvi[k - 1] * (Q[k] - Q[k - 1]))
        else:
            fds[k] = fdq[k] = zero
    dse, dqa = [None] * kx, [None] * kx
    dse[B], dqa[B] = fds[B] - fus[B], fdq[B] - fuq[B]
    fsum, precnv = zero, zero
    for k in range(B):
        on = k >= iptop
        dse[k] = torch.where(on, (fus[k + 1] - fds[k + 1]) - (fus[k] - fds[k]), zero)
        dqa[k] = torch.where(on, (fuq[k + 1] - fdq[k + 1]) - (fuq[k] - fdq[k]), zero)
        delq = torch.where(on, par["rhil"] * QS[k] - Q[k], zero)
        fsq = torch.where(delq > 0.0, par["smf"] * cbmf * delq, zero)
        dqa[k], fsum = dqa[k] + fsq, fsum + fsq
        top = iptop == k + 1
        qsatb = QS[k] + wvi[k] * (QS[k + 1] - QS[k])
        pr = _at_least(fuq[k + 1] - fm[k + 1] * qsatb, 0.0)
        precnv = torch.where(top, pr, precnv)
        dse[k] = torch.where(top, fus[k + 1] - fds[k + 1] + ALHC * pr, dse[k])
        dqa[k] = torch.where(top, fuq[k + 1] - fdq[k + 1] - pr, dqa[k])
    dqa[B] = dqa[B] - fsum
    DT[0], DQ[0] = dse[0], dqa[0]
    for k in range(1, kx):
        DT[k], DQ[k] = dse[k] / psa * V["grdscp"][k], dqa[k] / psa * V["grdsig"][k]
    # large-scale condensation
    rtl = 1.0 / (par["trlsc"] * 3600.0)
    psum, first = zero, torch.zeros_like(iptop)
    for k in range(kx - 1, 0, -1):
        s2 = fsg[k] * fsg[k]
        rhref = torch.maximum(par["rhlsc"] + par["drhlsc"] * (s2 - 1.0), par["rhblsc"])
        dqa_k = rhref * QS[k] - Q[k]
        wet = dqa_k < 0.0
        dql = torch.where(wet, dqa_k * rtl, zero)
        dtl = torch.where(wet, ALHC / CP * torch.minimum(-dqa_k * rtl, 10.0 * s2 * rtl * psa ** 2),
                          zero)
        first = torch.where(wet, k, first)
        DT[k], DQ[k] = DT[k] + dtl, DQ[k] + dql
        psum = psum + dhs[k] * P0 / GRAV * dql
    precls = -psum * psa
    iptop = torch.minimum(torch.where(first == 0, 1, first), iptop)
    # clouds
    N = kx - 2
    m0 = RH[N] > R["rhcl1"]
    cl0 = torch.where(m0, RH[N] - R["rhcl1"], zero)
    icl0 = torch.where(m0, N, kx)
    upd, iup, cmax = {}, {}, None
    for k in range(2, kx - 2):
        drh = RH[k] - R["rhcl1"]
        m = (drh > cl0) & (Q[k] > R["qacl"])
        upd[k], iup[k] = torch.where(m, drh, cl0), torch.where(m, k, icl0)
        cmax = upd[k] if cmax is None else torch.maximum(cmax, upd[k])
    icl = torch.full_like(icl0, -1)
    for k in range(2, kx - 2):
        icl = torch.maximum(icl, torch.where(cmax == upd[k], iup[k], icl0))
    icltop = torch.minimum(iptop, icl)
    if levels is None:
        return icltop.clamp(0, kx - 1)
    gse = (SE[N] - SE[B]) / (PHI[N] - PHI[B])
    pr1 = _at_most(86.4 * (precnv + precls), R["pmaxcl"])
    cloudc = _at_most(R["wpcl"] * torch.sqrt(_at_least(pr1, 1e-9))
                      + _at_most(cmax / (R["rhcl2"] - R["rhcl1"]), 1.0) ** 2, 1.0)
    fstab = _at_most(_at_least((gse - R["gse_s0"]) / (R["gse_s1"] - R["gse_s0"]), 0.0), 1.0)
    clstr = fstab * _at_least(R["clsmax"] - 1.2 * cloudc, 0.0)
    clstr = clstr + b["fmask"] * (_at_least(clstr, R["clsminl"]) * RH[B] - clstr)
    # shortwave
    snowc = torch.clamp(b["snowc"], max=1.0)
    alb_l = b["alb0"] + snowc * (R["albsn"] - b["alb0"])
    alb_s = R["albsea"] + b["sice"] * (R["albice"] - R["albsea"])
    albsfc = alb_s + b["fmask"] * (alb_l - alb_s)
    z = _solar(_single(80.0 / DAYS_YEAR), b["sia"], b["coa"])
    refl = torch.where(icltop < kx, par["albcl"] * cloudc, zero)
    r = [refl if levels[k] else zero for k in range(kx)]
    r[B] = par["albcls"] * clstr
    psaz = psa * z["zenit"]
    acloud = cloudc * _at_most(R["abscl1"] * Q[N], R["abscl2"])
    tau0, tau1 = [None] * kx, [None] * kx
    for k in range(kx):
        a = R["absdry"]
        if k > 0:
            a = a + R["absaer"] * fsg[k] * fsg[k] + R["abswv1"] * Q[k]
            tau1[k] = torch.exp(-psaz * dhs[k] * R["abswv2"] * Q[k])
        if 0 < k < B:
            a = a + torch.where(k >= icltop, acloud, zero)
        tau0[k] = torch.exp(-psaz * dhs[k] * a)
    heat = [zero] * kx
    f1 = z["fsol"] * 0.95
    g = tau0[0] * (f1 - z["ozupp"] * psa)
    heat[0], f1 = f1 - g, g
    g = tau0[1] * (f1 - z["ozone"] * psa)
    heat[1], f1 = f1 - g, g
    back = [r[0], r[1]]
    for k in range(2, kx):
        heat[k] = f1 * (1.0 - r[k]) * (1.0 - tau0[k])
        back.append(r[k] * f1)
        f1 = f1 * tau0[k] * (1.0 - r[k])
    f2 = z["fsol"] * 0.05
    for k in range(1, kx):
        heat[k] = heat[k] + f2 * (1.0 - tau1[k])
        f2 = f2 * tau1[k]
    rsds = f1 + f2
    up = f1 * albsfc
    rsns = rsds - up
    heat[B] = heat[B] + up * (1.0 - tau0[B])
    for k in range(B, 0, -1):
        up = up * tau0[k] + back[k]
        heat[k - 1] = heat[k - 1] + up * (1.0 - tau0[k - 1])
    fsw0, fsw1 = tau0[0] * up + r[0], f2
    ftop_sw = z["fsol"] - fsw0
    if step % 3 == 0:
        for k in range(kx):
            DT[k] = DT[k] + heat[k] * V["grdscp"][k] / psa
    # longwave: transmissivities, blackbody terms, downward pass
    acl1, acl2 = cloudc * R["ablcl1"], cloudc * R["ablcl2"]
    th = [T[k] + wvi[k] * (T[k + 1] - T[k]) for k in range(kx - 1)]
    tau, s0, s1, fb = [], [], [], []

    def fractions(t):
        j = _at_most(_at_least(t, 200.0), 320.0)
        f = [None, 0.148 - 3.0e-6 * (j - 247.0) ** 2, 0.356 - 5.2e-6 * (j - 282.0) ** 2,
             0.314 + 1.0e-5 * (j - 315.0) ** 2]
        f[0] = 1.0 - (f[1] + f[2] + f[3])
        return [(1.0 - R["epslw"]) * a for a in f]

    for k in range(kx):
        a = [R["ablwin"] + zero, R["ablco2"] + zero, R["ablwv1"] * Q[k], R["ablwv2"] * Q[k]]
        if k == 0:
            a[2] = a[3] = zero
        if 2 <= k <= kx - 2:
            a[0] = a[0] + torch.where(k > icltop, acl1, acl2)
            a[2], a[3] = torch.maximum(a[2], acl2), torch.maximum(a[3], acl2)
        tau.append([torch.exp(-v * psa * dhs[k]) for v in a])
        fb.append(fractions(T[k]))
        if k == 0:
            s0.append(SBC * (0.75 * T[0] + 0.25 * th[0]) ** 4)
            s1.append(zero)
        elif k == 1:
            s0.append(SBC * (0.5 * T[1] + 0.25 * (th[0] + th[1])) ** 4)
            s1.append(zero)
        else:
            grad = (0.5 * _at_least(th[k] - th[k - 1], 0.0) if k < B
                    else _at_least(T[B] - th[B - 1], 0.0))
            s0.append(SBC * T[k] ** 4)
            s1.append(4.0 * SBC * T[k] ** 3 * grad)
    div = [zero] * kx
    fl = [(1.0 - tau[0][i]) * fb[0][i] * (s0[0] + (1.0 - tau[0][i]) * s1[0]) if i < 2 else zero
          for i in range(4)]
    prev = sum(fl)
    div[0] = -prev
    for k in range(1, kx):
        fl = [tau[k][i] * fl[i] + (1.0 - tau[k][i]) * fb[k][i] * (s0[k] + (1.0 - tau[k][i]) * s1[k])
              for i in range(4)]
        cur = sum(fl)
        div[k] = prev - cur
        prev = cur
    corlw = R["epslw"] * R["emisfc"] * s0[B]
    div[B] = div[B] - corlw
    rlds = R["emisfc"] * prev + corlw
    # surface fluxes
    du = dv = tsfc = tskin_out = shf = evap = rlus = zero
    esbc = R["emisfc"] * SBC
    sst = b["sst"]
    if land:
        rdth = R["fstab"] / R["dtheta"]
        phi0 = b["orog"] * GRAV
        dt1 = wvi[B] * (T[B] - T[B - 1])
        t10 = T[B] + dt1
        t11 = t10 - phi0 * dt1 / (RGAS * 288.0 * V["sigl"][B])
        t21 = T[B] + PHI[B] / CP
        t20 = t21 - phi0 / CP
        warm = T[B] > T[B - 1]
        f0 = R["ftemp0"]
        t10 = torch.where(warm, f0 * t10 + (1.0 - f0) * t20, T[B])
        t11 = torch.where(warm, f0 * t11 + (1.0 - f0) * t21, T[B])
        t0 = t11 + b["fmask"] * (t10 - t11)
        wind = torch.sqrt((R["fwind0"] * x["u"]) ** 2 + (R["fwind0"] * x["v"]) ** 2
                          + R["vgust"] ** 2)
        denv = P0 * psa / (RGAS * t0) * wind

        def stable(d):
            return torch.where(d > 0.0, _at_most(d, R["dtheta"]), _at_least(0.5 * d, -R["dtheta"]))

        tskin = b["stl"] + R["ctday"] * torch.sqrt(b["coa"]) * rsds * (1.0 - alb_l) * psa
        denv1 = denv * (1.0 + stable(tskin - t20) * rdth)
        rhd = 1.0 / (GRAV * R["hdrag"])
        cdl = R["cdl"] * denv * (1.0 + rhd * (1.0 - torch.exp(-torch.clamp(b["phis0"], min=0.0)
                                                               * rhd)))
        shf0 = R["chl"] * CP * denv1 * (tskin - t10)
        qs0 = _qsat(tskin, psa, 1.0)
        evap0 = R["chl"] * denv1 * _at_least(b["soilw"] * qs0 - Q[B], 0.0)
        drls, rlus0 = 4.0 * esbc * tskin ** 3, esbc * tskin ** 4
        clamb = R["clambda"] + snowc * (R["clambsn"] - R["clambda"])
        hfl = (rsds * (1.0 - alb_l) + rlds - (rlus0 + shf0 + ALHC * evap0)
               - clamb * (tskin - b["stl"]))
        dqs = torch.where(evap0 > 0.0, b["soilw"] * (_qsat(tskin + 1.0, psa, 1.0) - qs0), zero)
        dts = hfl / (clamb + drls + R["chl"] * denv1 * (CP + ALHC * dqs))
        tskin = tskin + dts
        shf0, evap0 = shf0 + R["chl"] * CP * denv1 * dts, evap0 + R["chl"] * denv1 * dqs * dts
        rlus0 = rlus0 + drls * dts
        denv2 = denv * (1.0 + stable(sst - t21) * rdth)
        cds = R["cds"] * denv2
        shf1 = R["chs"] * CP * denv2 * (sst - t11)
        evap1 = R["chs"] * denv2 * (_qsat(sst, psa, 1.0) - Q[B])
        rlus1 = esbc * sst ** 4
        mix = lambda sea, lnd: sea + b["fmask"] * (lnd - sea)
        du = mix(-cds * x["u"], -cdl * x["u"]) / psa * V["grdsig"][B]
        dv = mix(-cds * x["v"], -cdl * x["v"]) / psa * V["grdsig"][B]
        shf, evap, rlus = mix(shf1, shf0), mix(evap1, evap0), mix(rlus1, rlus0)
        tsfc, tskin_out = mix(sst, b["stl"]), mix(sst, tskin)
        DT[B] = DT[B] + shf / psa * V["grdscp"][B]
        DQ[B] = DQ[B] + evap / psa * V["grdsig"][B]
    # longwave: upward pass
    rlns = rlus - rlds
    ref = 1.0 - R["emisfc"]
    fs = fractions(tsfc)
    fl = [fs[0] * rlus + ref * fsw0, fs[1] * rlus + ref * fsw1, fs[2] * rlus, fs[3] * rlus]
    div[B] = div[B] + R["epslw"] * rlus
    prev = sum(fl)
    for k in range(B, 0, -1):
        fl = [tau[k][i] * fl[i] + (1.0 - tau[k][i]) * fb[k][i] * (s0[k] - (1.0 - tau[k][i]) * s1[k])
              for i in range(4)]
        cur = sum(fl)
        div[k] = div[k] + prev - cur
        prev = cur
    top = [tau[0][i] * fl[i] + (1.0 - tau[0][i]) * fb[0][i] * s0[0] for i in range(2)]
    strat = R["epslw"] / (dhs[0] + dhs[1]) * psa
    cor1, cor2 = dhs[0] * strat * s0[0] + z["stratz"] * psa, dhs[1] * strat * s0[1]
    div[0] = div[0] + (fl[0] - top[0]) + (fl[1] - top[1]) - cor1
    div[1] = div[1] - cor2
    ftop_lw = cor1 + cor2 + top[0] + top[1] + fl[2] + fl[3]
    for k in range(kx):
        DT[k] = DT[k] + div[k] * V["grdscp"][k] / psa
    # vertical diffusion
    cshc = dhs[B] / 3600.0
    cvdi = (hsg[B] - hsg[1]) / ((B - 1) * 3600.0)
    fvdiq, fvdise = cvdi / R["trvdi"], cvdi / (R["trvds"] * CP)
    dmse = SE[B] - SE[B - 1] + ALHC * (Q[B] - QS[B - 1])
    drh = RH[B] - RH[B - 1]
    fcnv = torch.where((kx - iptop - 1 > 0) & (dmse >= 0.0), R["redshc"], 1.0)
    fse = torch.where(dmse >= 0.0, fcnv * cshc / (R["trshc"] * CP) * dmse, zero)
    fq = torch.where((dmse >= 0.0) & (drh >= 0.0), fcnv * cshc / R["trshc"] * QS[B] * drh,
                     torch.where((dmse < 0.0) & (drh > R["rhgrad"] * (fsg[B] - fsg[B - 1])),
                                 fvdiq * hsg[B] * QS[B - 1] * drh, zero))
    DT[B - 1], DT[B] = DT[B - 1] + fse / dhs[B - 1], DT[B] - fse / dhs[B]
    DQ[B - 1], DQ[B] = DQ[B - 1] + fq / dhs[B - 1], DQ[B] - fq / dhs[B]
    for k in range(2, kx - 2):
        if _single(hsg[k + 1]) > 0.5:
            d = RH[k + 1] - RH[k]
            f = torch.where(d >= R["rhgrad"] * (fsg[k + 1] - fsg[k]),
                            fvdiq * hsg[k + 1] * QS[k] * d, zero)
            DQ[k], DQ[k + 1] = DQ[k] + f / dhs[k], DQ[k + 1] - f / dhs[k + 1]
    cum = zero
    for k in range(B):
        se0 = SE[k + 1] - R["segrad"] * (PHI[k + 1] - PHI[k])
        f = torch.where(SE[k] < se0, fvdise * (se0 - SE[k]), zero)
        cum = cum + f / (1.0 - hsg[k + 1])
        DT[k], DT[k + 1] = DT[k] + f / dhs[k], DT[k + 1] - cum
    if verify:
        DQ = [torch.where(Qraw[k] + dt_seconds * DQ[k] >= 0.0, DQ[k], -Qraw[k] / dt_seconds)
              for k in range(kx)]
    return dict(du=du, dv=dv, t=DT, q=DQ, precnv=precnv, precls=precls, iptop=iptop,
                icltop=icltop, cbmf=cbmf, cloudc=cloudc, cloudstr=clstr, rsds=rsds, rsns=rsns,
                ftop_sw=ftop_sw, rlds=rlds, rlns=rlns, ftop_lw=ftop_lw, tsfc=tsfc,
                tskin=tskin_out, shf=shf, evap=evap)


class _Grid:
    """Float64 columns of one grid, evaluated in chunks."""

    def __init__(self, f, kx, ix, il, land, verify):
        self.kx, self.n, self.land, self.verify = kx, ix * il, land, verify
        d = lambda a: a.double().reshape(-1, self.n) if a.dim() == 3 else a.double().reshape(-1)
        lat = lambda a: a.double()[None, :].expand(ix, il).reshape(-1)
        self.x = dict(u=d(f["u"])[-1], v=d(f["v"])[-1], t=d(f["t"]), q=d(f["q"]),
                      phi=d(f["phi"]), psa=d(f["psa"]))
        self.b = {k: d(f[k]) for k in ("sst", "stl", "soilw", "snowc", "sice", "alb0", "fmask",
                                       "orog", "phis0")}
        self.b.update(sia=lat(f["sia"]), coa=lat(f["coa"]))
        self.par = {k: torch.tensor(_single(v), dtype=torch.float64, device=f["psa"].device)
                    for k, v in _P.items()}

    def _eval(self, x, par, a, z, step, levels):
        return _physics(x, {k: v[a:z] for k, v in self.b.items()}, par, self.kx, self.land,
                        self.verify, 1800.0, step, levels)

    def _cut(self, x, a, z):
        return {k: list(v[:, a:z].unbind(0)) if v.dim() == 2 else v[a:z] for k, v in x.items()}

    def _chunks(self):
        return [(a, min(a + CHUNK, self.n)) for a in range(0, self.n, CHUNK)]

    def levels(self, x):
        """Whether level k is any column's cloud top."""
        hit = torch.zeros(self.kx, dtype=torch.bool, device=x["psa"].device)
        with torch.no_grad():
            for a, z in self._chunks():
                top = self._eval(self._cut(x, a, z), self.par, a, z, 0, None)
                hit |= torch.bincount(top, minlength=self.kx) > 0
        return hit.tolist()

    def forward(self, x, step=0):
        """{field: [n] or [kx, n]} of the tendencies and diagnostics."""
        levels, parts = self.levels(x), []
        with torch.no_grad():
            for a, z in self._chunks():
                o = self._eval(self._cut(x, a, z), self.par, a, z, step, levels)
                parts.append({k: torch.stack(v) if isinstance(v, list) else v
                              for k, v in o.items()})
        return {k: torch.cat([p[k] for p in parts], -1) for k in parts[0]}

    def vjp(self, x, ct, step=0):
        """Gradients of <ct, tendencies>: the state's as [n] or [kx, n], and the parameters'."""
        levels = self.levels(x)
        grad, total = {k: [] for k in x}, torch.zeros(len(PARAMS), dtype=torch.float64,
                                                      device=x["psa"].device)
        for a, z in self._chunks():
            xc = self._cut(x, a, z)
            xc = {k: [t.clone().requires_grad_() for t in v] if isinstance(v, list)
                  else v.clone().requires_grad_() for k, v in xc.items()}
            par = {k: v.clone().requires_grad_() for k, v in self.par.items()}
            o = self._eval(xc, par, a, z, step, levels)
            loss = (o["du"] * ct["u"][a:z] + o["dv"] * ct["v"][a:z]).sum()
            for k in range(self.kx):
                loss = loss + (o["t"][k] * ct["t"][k, a:z] + o["q"][k] * ct["q"][k, a:z]).sum()
            flat = [t for v in xc.values() for t in (v if isinstance(v, list) else [v])]
            got = iter(torch.autograd.grad(loss, flat + list(par.values()), allow_unused=True))
            new = lambda t, g: torch.zeros_like(t) if g is None else g
            for k, v in xc.items():
                grad[k].append(torch.stack([new(t, next(got)) for t in v])
                               if isinstance(v, list) else new(v, next(got)))
            total += torch.stack([new(v, next(got)) for v in par.values()])
        return {k: torch.cat(v, -1) for k, v in grad.items()}, total


def _dense(low, kx):
    """A lowest-level plane as the dense level field whose other levels are zero."""
    out = torch.zeros(kx, low.numel(), dtype=low.dtype, device=low.device)
    out[-1] = low
    return out


def _exact_call(f, kx, ix, il, land, verify):
    grid = _Grid(f, kx, ix, il, land, verify)
    o = grid.forward(grid.x)
    s3 = lambda a: a.reshape(kx, ix, il)
    out = dict(u=s3(_dense(o["du"], kx)), v=s3(_dense(o["dv"], kx)), t=s3(o["t"]), q=s3(o["q"]))
    out.update({k: v.reshape(ix, il) for k, v in o.items() if k not in ("du", "dv", "t", "q")})
    out["iptop"] = out["icltop"] = None
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        members = _members(case["scale"])
        at, n3, n2 = _ensemble_offsets(members)
        flat = {k: torch.zeros(n2 if k in ("precnv", "precls") else n3, device=_device(),
                               dtype=torch.float64) for k in ENS_FIELDS}
        for i, ((ix, il, kx), (o3, o2)) in enumerate(zip(members, at)):
            o = _exact_call(_fields(seed * 1000 + i, ix, il, kx), kx, ix, il, True, False)
            for k, name in zip(("u", "v", "t", "q", "precnv", "precls"), ENS_FIELDS):
                at0 = o2 if k in ("precnv", "precls") else o3
                flat[name][at0:at0 + o[k].numel()] = o[k].reshape(-1)
        return flat
    kx, ix, il = case["kx"], case["ix"], case["il"]
    land, verify = case.get("land", True), case.get("verify", False)
    f = _fields(seed, ix, il, kx, land, verify)
    if kind == "hs":
        return _exact_hs(f, kx, il)
    if kind == "call":
        o = _exact_call(f, kx, ix, il, land, verify)
        names = ("u", "v", "t", "q", "precnv", "precls")
        return o if case["diag"] else {k: o[k] for k in names}
    s3, s2 = (lambda a: a.reshape(kx, ix, il)), (lambda a: a.reshape(ix, il))
    whole = lambda g: dict(u=s3(_dense(g["u"], kx)), v=s3(_dense(g["v"], kx)), t=s3(g["t"]),
                           q=s3(g["q"]), phi=s3(g["phi"]), psa=s2(g["psa"]))
    ct = {k: v.double().reshape(kx, -1) for k, v in _cotangent(seed, kx, ix, il).items()}
    grid = _Grid(f, kx, ix, il, land, verify or kind == "rollout")
    if kind == "vjp":
        g, p = grid.vjp(grid.x, dict(u=ct["u"][-1], v=ct["v"][-1], t=ct["t"], q=ct["q"]))
        return dict(whole(g), params=p)
    # rollout: x_{n+1} = x_n + dt f_n(x_n), then the steps' gradients last to first
    dt, xs = 1800.0, [grid.x]
    for n in range(case["nsteps"]):
        o, x = grid.forward(xs[-1], n), xs[-1]
        xs.append(dict(x, u=x["u"] + dt * o["du"], v=x["v"] + dt * o["dv"],
                       t=x["t"] + dt * o["t"], q=x["q"] + dt * o["q"]))
    bar = dict(u=ct["u"][-1], v=ct["v"][-1], t=ct["t"], q=ct["q"])
    fixed = dict(phi=torch.zeros_like(ct["t"]), psa=torch.zeros_like(grid.x["psa"]))
    par = torch.zeros(len(PARAMS), dtype=torch.float64, device=_device())
    for n in reversed(range(case["nsteps"])):
        g, p = grid.vjp(xs[n], {k: dt * v for k, v in bar.items()}, n)
        bar = {k: bar[k] + g[k] for k in bar}
        fixed = {k: fixed[k] + g[k] for k in fixed}
        par = par + p
    wind = lambda a, low: torch.cat([a.double().reshape(kx, -1)[:-1], low[None]], 0)
    grad = dict(whole(dict(bar, **fixed)), u=s3(wind(ct["u"], bar["u"])),
                v=s3(wind(ct["v"], bar["v"])))
    last = dict(u=s3(wind(f["u"], xs[-1]["u"])), v=s3(wind(f["v"], xs[-1]["v"])),
                t=s3(xs[-1]["t"]), q=s3(xs[-1]["q"]))
    return dict(final=last, grad=grad, params=par)


def _exact_hs(f, kx, il):
    day, sigma_b = 86400.0, _single(0.7)
    kf, ka, ks = (_single(v) for v in (1.0 / day, 1.0 / (40 * day), 1.0 / (4 * day)))
    la = torch.as_tensor(_latitudes(il), device=f["t"].device)
    s2, c2, c4 = torch.sin(la) ** 2, torch.cos(la) ** 2, torch.cos(la) ** 4
    sig = torch.as_tensor(_vertical(kx)["fsg"], device=f["t"].device).double()[:, None, None]
    p = sig * f["psa"].double()
    teq = torch.clamp(p ** _single(2.0 / 7.0) * (315.0 - 60.0 * s2 - 10.0 * torch.log(p) * c2),
                      min=200.0)
    cut = torch.clamp((sig - sigma_b) / (1.0 - sigma_b), min=0.0)
    t = f["t"].double()
    return dict(u=-kf * cut * f["u"].double(), v=-kf * cut * f["v"].double(),
                t=-(ka + (ks - ka) * cut * c4) * (t - teq), q=torch.zeros_like(t))
