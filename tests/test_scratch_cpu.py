"""The forward's scratch (the level-set prediction of the last call): one per stream and thread, kept
from call to call (a captured graph holds its address)."""
import importlib
import threading

import pytest
import torch

pkg = importlib.import_module("jax-gcm_b200")
physics = importlib.import_module("jax-gcm_b200.physics")


@pytest.fixture
def scratch(monkeypatch):
    inst = pkg.synthetic.land_instance(3, 4, 2, 8)
    st, fo, ge, da = pkg.instance_to_device(inst, "cpu")
    phys = pkg.SpeedyPhysics()
    desc = phys.desc(ge, da, True)

    def on(stream):
        monkeypatch.setattr(physics, "current_raw_stream", lambda index: stream)
        return phys._scratch_for(desc, torch.device("cpu"))

    monkeypatch.setattr(physics, "current_raw_stream", lambda index: 0)
    on.physics = phys
    return on


def test_streams_do_not_share(scratch):
    a, b = scratch(11), scratch(12)
    assert a.data_ptr() != b.data_ptr()
    assert scratch(11) is a and scratch(12) is b


def test_threads_do_not_share(scratch):
    mine, other = scratch(11), []
    t = threading.Thread(target=lambda: other.append(scratch(11)))
    t.start()
    t.join()
    assert other[0].data_ptr() != mine.data_ptr() and scratch(11) is mine


def test_no_scratch_is_kept_for_an_empty_grid(scratch):
    from types import SimpleNamespace
    desc = scratch.physics.desc(SimpleNamespace(nodal_shape=(8, 4, 0)), SimpleNamespace(
        dt_seconds=1.0, tyear=0.0, model_year=1950, model_step=0), True)
    assert scratch.physics._scratch_for(desc, torch.device("cpu")).numel() == 0
    assert scratch(0).numel() > 0
