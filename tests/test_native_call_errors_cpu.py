"""Errors of the native calls arrive as Python exceptions: a wrong argument count, a field that is no
tensor, a missing attribute, an object that is no address.  In a child process, since an exception
that does not find its way out of the extension module ends the interpreter."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHILD = """
import importlib
pkg = importlib.import_module("jax-gcm_b200")
calls = pkg._lib.calls()
inst = pkg.synthetic.land_instance(3, 4, 2, 8)

def error(name, *args):
    try:
        getattr(calls, name)(*args)
    except Exception as e:
        print(name, type(e).__name__)
    else:
        print(name, "none")

for name in ("fwd", "vjp", "held_suarez", "rollout_step", "rollout_reverse", "bind"):
    error(name, 1)
st, fo, ge, da = pkg.instance_to_device(inst, "cpu")
st.temperature = 3
error("fwd", st, fo, ge, None, True, 64, 64, 64, 64, 64, 0)
error("vjp", st, fo, ge, st, 64, 64, 64, 64)
error("held_suarez", st, st.u_wind, None, 64)
del st.u_wind
error("rollout_step", st, st, 1.0)
error("bind", "a", "b", "c", "d", "e")
"""
WANT = ["fwd TypeError", "vjp TypeError", "held_suarez TypeError", "rollout_step TypeError",
        "rollout_reverse TypeError", "bind TypeError", "fwd TypeError", "vjp TypeError",
        "held_suarez TypeError", "rollout_step AttributeError", "bind TypeError"]


def test_errors_are_python_exceptions():
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.split("\n")[:-1] == WANT
