"""What the rollout's kernels leave to torch's own operations: planes that are more than their values
in memory."""
import importlib

import pytest

pytestmark = pytest.mark.gpu
EVOLVED = ("u_wind", "v_wind", "temperature", "specific_humidity")


@pytest.fixture(scope="module")
def case():
    pkg = importlib.import_module("jax-gcm_b200")
    return pkg, pkg.instance_to_device(pkg.synthetic.land_instance(3, 12, 6, 8), "cuda")


def test_forward_mode_tangents_travel(case):
    import torch
    import torch.autograd.forward_ad as fw
    pkg, (st, fo, ge, da) = case
    phys = pkg.SpeedyPhysics(fuse_verify=True, time_step=1800.0, diagnostics=False)
    want = pkg.rollout.step(phys, st, fo, ge, da, 1800.0)
    tangent = torch.randn_like(st.temperature)
    with fw.dual_level():
        dual = st.copy(temperature=fw.make_dual(st.temperature, tangent))
        got = fw.unpack_dual(pkg.rollout.step(phys, dual, fo, ge, da, 1800.0).temperature)
        assert torch.equal(got.primal, want.temperature)
        # the physics carries none: x + dt f passes x's on
        assert got.tangent is not None and torch.equal(got.tangent, tangent)


def test_other_tensors_take_the_general_path(case):
    import torch
    from torch.utils._python_dispatch import TorchDispatchMode
    pkg, (st, fo, ge, da) = case
    calls = pkg._lib.calls()
    x = [getattr(st, k) for k in EVOLVED]
    f = [torch.randn_like(t) for t in x]

    class Sub(torch.Tensor):
        pass

    class Watch(TorchDispatchMode):
        seen = 0

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            Watch.seen += 1
            return func(*args, **(kwargs or {}))

    assert calls.rollout_step(x, f, 1.0) is not None
    assert calls.rollout_step([torch._neg_view(t) for t in x], f, 1.0) is None
    assert calls.rollout_step([t.as_subclass(Sub) for t in x], f, 1.0) is None
    with Watch():
        assert calls.rollout_step(x, f, 1.0) is None
        phys = pkg.SpeedyPhysics(fuse_verify=True, time_step=1800.0, diagnostics=False)
        pkg.rollout.step(phys, st, fo, ge, da, 1800.0)
    assert Watch.seen > 0
