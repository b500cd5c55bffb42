"""Calls that overlap on two streams give the bits of the same calls one after the other."""
import importlib
from dataclasses import replace

import pytest

pytestmark = pytest.mark.gpu
STATE = ("u_wind", "v_wind", "temperature", "specific_humidity", "geopotential",
         "normalized_surface_pressure")


@pytest.fixture(scope="module")
def pkg():
    return importlib.import_module("jax-gcm_b200")


def instances(pkg):
    """Two instances of one size whose dates, solar rows and level sets differ."""
    import torch
    out = []
    for i in range(2):
        inst = pkg.synthetic.land_instance(40 + i, 96, 48, 8)
        if i:
            inst.q[:5, ::7] *= 5.0
        st, fo, ge, da = pkg.instance_to_device(inst, "cuda")
        gen = torch.Generator(device="cuda").manual_seed(i)
        ct = pkg.PhysicsTendency(*(torch.randn(8, 96, 48, generator=gen, device="cuda")
                                   for _ in range(4)))
        out.append((st, fo, ge, replace(da, tyear=0.1 + 0.5 * i), ct))
    return out


def test_vjps_on_two_streams(pkg):
    import torch
    phys = pkg.SpeedyPhysics(diagnostics=False)
    cases = instances(pkg)
    call = lambda c: pkg.adjoint.vjp(phys, *c)[0]
    want = [call(c) for c in cases]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in cases]
    got = []
    for _ in range(20):
        for c, s in zip(cases, streams):
            with torch.cuda.stream(s):
                got.append(call(c))
    torch.cuda.synchronize()
    for i, g in enumerate(got):
        for n in STATE:
            assert torch.equal(getattr(g, n), getattr(want[i % 2], n)), (i, n)


def test_forwards_of_one_object_on_two_streams(pkg):
    import torch
    cases = [c[:4] for c in instances(pkg)]
    out = lambda r: [getattr(r[0], n) for n in STATE[:4]] + [r[1].condensation.precls]
    want = [out(pkg.SpeedyPhysics(speculate=False).compute_tendencies(*c)) for c in cases]
    torch.cuda.synchronize()
    phys = pkg.SpeedyPhysics()
    streams = [torch.cuda.Stream() for _ in cases]
    got = []
    for _ in range(20):
        for c, s in zip(cases, streams):
            with torch.cuda.stream(s):
                got.append(out(phys.compute_tendencies(*c)))
    torch.cuda.synchronize()
    for i, g in enumerate(got):
        assert all(torch.equal(a, b) for a, b in zip(g, want[i % 2])), i


def test_forwards_of_one_object_from_two_threads(pkg):
    """Two threads on one stream, whose calls' launches may interleave."""
    import threading

    import torch
    cases = [c[:4] for c in instances(pkg)]
    out = lambda r: [getattr(r[0], n) for n in STATE[:4]] + [r[1].condensation.precls]
    want = [out(pkg.SpeedyPhysics(speculate=False).compute_tendencies(*c)) for c in cases]
    phys, got = pkg.SpeedyPhysics(), [[], []]

    def work(i):
        for _ in range(50):
            got[i].append(out(phys.compute_tendencies(*cases[i])))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for i in range(2):
        assert len(got[i]) == 50
        for g in got[i]:
            assert all(torch.equal(a, b) for a, b in zip(g, want[i])), i


@pytest.mark.parametrize("warm", [False, True])
def test_captured_calls(pkg, warm):
    """A forward and a VJP captured on the graph's own stream, without and with calls before it on
    another, while the object goes on being called; two graphs of one object."""
    import torch
    cases = instances(pkg)
    phys = pkg.SpeedyPhysics(diagnostics=False)
    if warm:
        phys.compute_tendencies(*cases[0][:4])
    pkg._lib.preload(0)
    want = [([getattr(pkg.SpeedyPhysics(speculate=False).compute_tendencies(*c[:4])[0], n)
              for n in STATE[:4]], pkg.adjoint.vjp(phys, *c)[0]) for c in cases]
    torch.cuda.synchronize()
    graphs = []
    for c in cases:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            tend, _ = phys.compute_tendencies(*c[:4])
            grad, _ = pkg.adjoint.vjp(phys, *c)
        graphs.append((g, tend, grad))
    for i in range(6):
        (g, tend, grad), (wt, wg) = graphs[i % 2], want[i % 2]
        g.replay()
        phys.compute_tendencies(*cases[1 - i % 2][:4])
        torch.cuda.synchronize()
        assert all(torch.equal(getattr(tend, n), w) for n, w in zip(STATE[:4], wt)), i
        assert all(torch.equal(getattr(grad, n), getattr(wg, n)) for n in STATE), i
