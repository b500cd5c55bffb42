"""A member's results do not depend on the batch that carries it: members that fuse verify and members
that do not, in one launch, against each member alone, in every bit; and the adjoint's register
budgets without verify (tests/test_adjoint_tiles_gpu.py has them with it).  A launch without a
verifying class takes the forms built without verify, one with such a class the others, and the
member count and size choose the register budget."""
import ctypes as C
import importlib

import pytest

pytestmark = pytest.mark.gpu
LEVELS = ("u_wind", "v_wind", "temperature", "specific_humidity")
STATE = LEVELS + ("geopotential", "normalized_surface_pressure")
SMALL, LARGE = [(43, 3), (16, 8)], [(43, 3), (300, 256)]


@pytest.fixture(scope="module")
def pkg():
    return importlib.import_module("jax-gcm_b200")


class Batch:
    """One class per (level count, verify); one member per class and grid."""

    def __init__(self, pkg, levels, grids):
        import torch
        self.pkg, self.L, self.cases = pkg, pkg._lib, []
        kinds = [(kx, v) for kx in levels for v in (False, True)]
        self.classes = (self.L.Class * len(kinds))()
        for i, (kx, verify) in enumerate(kinds):
            phys = pkg.SpeedyPhysics(diagnostics=False, fuse_verify=verify, time_step=1800.0)
            for ix, il in grids:
                inst = pkg.synthetic.land_instance(100 * kx + ix, ix, il, kx)
                inst.q[:, ::5] *= -0.3  # what verify_state clamps
                st, fo, ge, da = pkg.instance_to_device(inst, "cuda")
                gen = torch.Generator(device="cuda").manual_seed(ix)
                ct = pkg.PhysicsTendency(*(torch.randn(kx, ix, il, generator=gen, device="cuda")
                                           for _ in range(4)))
                self.cases.append((phys, st, fo, ge, da, ct, i))
            self.classes[i].desc = phys.desc(ge, da, True)
            self.classes[i].vgrid = ge.vgrid()
            self.classes[i].params = phys._pstruct

    def inputs(self, case):
        owner = lambda n: next(o for o in case[1:4] if hasattr(o, n))
        return self.L.Inputs(*[getattr(owner(n), n).data_ptr() for n in self.L.INPUT_FIELDS])

    def run(self, Member, fill, plan_bytes, plan, launch):
        import torch
        n = len(self.cases)
        mem, out = (Member * n)(), []
        for i, case in enumerate(self.cases):
            out.append(fill(mem[i], case))
            mem[i].inp = self.inputs(case)
            mem[i].ix, mem[i].il = case[3].nodal_shape[1:]
            mem[i].cls = case[6]
        nbytes = plan_bytes(mem, n)
        dev = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        host, info = (C.c_ubyte * nbytes)(), self.L.PlanInfo()
        nc = len(self.classes)
        assert plan(self.classes, nc, mem, n, C.cast(host, C.c_void_p),
                    C.c_void_p(dev.data_ptr()), nbytes, C.byref(info)) == 0
        dev.copy_(torch.frombuffer(bytearray(host), dtype=torch.uint8))
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert launch(self.classes, nc, C.c_void_p(dev.data_ptr()), C.byref(info), 0, stream) == 0
        torch.cuda.synchronize()
        return out


@pytest.mark.parametrize("levels,grids", [((8, 16), SMALL), ((8, 16), LARGE), ((7, 8), LARGE)])
def test_adjoint_members_with_and_without_verify(pkg, levels, grids):
    import torch
    b = Batch(pkg, levels, grids)
    lib = b.L.load()

    def fill(m, case):
        st, ct = case[1], case[5]
        g = [torch.empty_like(getattr(st, n)) for n in STATE] + [torch.empty(12, device="cuda")]
        m.ct = b.L.Cotangents(*[getattr(ct, n).data_ptr() for n in LEVELS])
        m.grads = b.L.Grads(*[t.data_ptr() for t in g])
        return g

    got = b.run(b.L.VjpMember, fill, lib.spd_ensemble_vjp_plan_bytes, lib.spd_ensemble_vjp_plan,
                lib.spd_ensemble_vjp)
    for g, (phys, st, fo, ge, da, ct, cls) in zip(got, b.cases):
        want, _ = pkg.adjoint.vjp(phys, st, fo, ge, da, ct)
        for n, t in zip(STATE, g):
            assert torch.equal(t, getattr(want, n)), (cls, ge.nodal_shape, n)


@pytest.mark.parametrize("levels,grids", [((8, 16), SMALL), ((8, 16), LARGE), ((7, 8), LARGE)])
def test_forward_members_with_and_without_verify(pkg, levels, grids):
    import torch
    b = Batch(pkg, levels, grids)
    lib = b.L.load()

    def fill(m, case):
        st = case[1]
        o = [torch.empty_like(getattr(st, n)) for n in LEVELS]
        o += [torch.empty_like(st.normalized_surface_pressure) for _ in range(2)]
        m.out = b.L.Outputs(*[t.data_ptr() for t in o])
        return o

    got = b.run(b.L.Member, fill, lib.spd_ensemble_plan_bytes, lib.spd_ensemble_plan,
                lib.spd_ensemble_fwd)
    for o, (phys, st, fo, ge, da, ct, cls) in zip(got, b.cases):
        tend, data = phys.compute_tendencies(st, fo, ge, da)
        want = [getattr(tend, n) for n in LEVELS] + [data.convection.precnv, data.condensation.precls]
        for i, (x, y) in enumerate(zip(o, want)):
            assert torch.equal(x, y), (cls, ge.nodal_shape, i)


@pytest.mark.parametrize("kx", [7, 8, 16])
def test_adjoint_register_budgets_without_verify(pkg, kx):
    """16,384 columns run two warps per scheduler, the 65,536 columns that contain them three or
    four."""
    import torch
    inst = pkg.synthetic.land_instance(77, 256, 256, kx)
    st, fo, ge, da = pkg.instance_to_device(inst, "cuda")
    phys = pkg.SpeedyPhysics(diagnostics=False)
    ct = [torch.randn(kx, 256, 256, device="cuda") for _ in range(4)]
    whole, _ = pkg.adjoint.vjp(phys, st, fo, ge, da, pkg.PhysicsTendency(*ct))
    cut = lambda t: t[..., :64, :].contiguous()
    part_of = lambda o, names: [cut(getattr(o, n)) for n in names]
    fo2 = pkg.ForcingData(*part_of(fo, ("alb0", "sice_am", "snowc_am", "soilw_am", "stl_am",
                                        "sea_surface_temperature")), lfluxland=fo.lfluxland)
    ge2 = pkg.Geometry.from_grid_shape((64, 256), kx, latitudes=inst.lat, device="cuda")
    ge2.orog, ge2.phis0, ge2.fmask = part_of(ge, ("orog", "phis0", "fmask"))
    ge2.sia, ge2.coa = ge.sia, ge.coa
    part, _ = pkg.adjoint.vjp(phys, pkg.PhysicsState(*part_of(st, STATE)), fo2, ge2, da,
                              pkg.PhysicsTendency(*map(cut, ct)))
    for n in STATE:
        assert torch.equal(getattr(part, n), cut(getattr(whole, n))), n
