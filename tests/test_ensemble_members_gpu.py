"""Ensembles whose member count passes the threads of the launches that walk the member list (the
one-block start of a call, the fixup's comparison): every member equal to the plain call bit for
bit, on the first call (every prediction misses) and on the next (every one holds)."""
import importlib

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 128, 129, 300])
def test_many_members_predict_and_redo(n):
    import torch
    pkg = importlib.import_module("jax-gcm_b200")
    insts = [pkg.synthetic.land_instance(9000 + i, 8, 5, (7, 8, 16)[i % 3]) for i in range(6)]
    objs = [pkg.instance_to_device(i, "cuda") for i in insts]
    date = objs[0][3]
    plain = []
    for st, fo, ge, da in objs:
        phys = pkg.SpeedyPhysics(diagnostics=False)
        plain.append(phys.compute_tendencies(st, fo, ge, date)[0])
    ens = pkg.Ensemble([pkg.Member(*objs[i % 6][:3]) for i in range(n)], date)
    for call in range(2):
        for m in ens.members:
            for t in m.out.values():
                t.fill_(float("nan"))
        out = ens.forward()
        torch.cuda.synchronize()
        for i, o in enumerate(out):
            for k in ("u_wind", "v_wind", "temperature", "specific_humidity"):
                assert torch.equal(o[k], getattr(plain[i % 6], k)), (n, call, i, k)
        assert ens.redone() == n
