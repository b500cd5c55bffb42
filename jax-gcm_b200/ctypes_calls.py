"""The native calls of ``csrc/torch_calls.cpp`` through ctypes: the same arguments, checks and results,
for an installation whose torch the extension module has not been built for (``_lib.calls``).
Slower on small calls by the 25 to 50 us that the extension module saves.
"""
from __future__ import annotations

import ctypes as C

import torch

from . import _lib
from ._lib import INPUT_FIELDS, OUTPUT_FIELDS

LEVELS = ("u_wind", "v_wind", "temperature", "specific_humidity")
STATE = INPUT_FIELDS[:6]
FORCING = INPUT_FIELDS[6:12]


def _values(t, need, name):
    if not isinstance(t, torch.Tensor):
        raise TypeError(f"{name} must be a tensor")
    if t.numel() < need:
        raise ValueError(f"{name} has {t.numel()} values, the geometry has {need}")
    return t


def _room(t, need, name):
    room = t.untyped_storage().nbytes() - t.storage_offset() * t.element_size()
    if room < 4 * need:
        raise ValueError(f"{name} (out) has room for {room // 4} values, the geometry has {need}")


def _on_device(device, outs=()):
    if device.type != "cuda":
        raise RuntimeError("the physics runs on CUDA tensors only (no CPU path)")
    if not all(t.is_cuda or t.is_pinned() for t in outs if t is not None):
        raise RuntimeError("out holds CUDA tensors")


def _inputs(state, forcing, geometry, desc, low_winds):
    """Contiguous float32 fields on the state's device, in spd_inputs_t's order."""
    columns = desc.ix * desc.il
    device = state.temperature.device
    fields = []
    for name in INPUT_FIELDS:
        owner = state if name in STATE else forcing if name in FORCING else geometry
        need = (desc.il if name in ("sia", "coa") else
                columns if low_winds and name in ("u_wind", "v_wind") else
                desc.kx * columns if name in LEVELS or name == "geopotential" else columns)
        fields.append(_values(getattr(owner, name), need, name))
    return device, [t.to(device=device, dtype=torch.float32).contiguous() for t in fields]


def _stream(device):
    return C.c_void_p(torch.cuda.current_stream(device).cuda_stream)


def _pointers(struct, tensors):
    return struct(*[None if t is None else t.data_ptr() for t in tensors])


def fwd(state, forcing, geometry, out, diagnostics, desc, vgrid, params, scratch, scratch_bytes,
        event):
    d = _lib.Desc.from_address(desc)
    low = bool(d.flags & _lib.SPD_LOW_LEVEL_WINDS)
    device, fields = _inputs(state, forcing, geometry, d, low)
    columns = d.ix * d.il
    if out is not None:
        for name, t in zip(OUTPUT_FIELDS, out):
            if t is not None:
                _room(t, d.kx * columns if name in LEVELS and not (low and name in LEVELS[:2])
                      else columns, name)
    _on_device(device, out or ())
    if out is None:
        names = OUTPUT_FIELDS if diagnostics else OUTPUT_FIELDS[:6]
        out = [torch.empty((d.kx, d.ix, d.il) if n in LEVELS else (d.ix, d.il), device=device,
                           dtype=torch.int32 if n in ("iptop", "icltop") else torch.float32)
               for n in names] + [None] * (len(OUTPUT_FIELDS) - len(names))
    rc = _lib.load().spd_fwd_marked(
        C.byref(d), C.byref(_lib.VGrid.from_address(vgrid)),
        C.byref(_lib.Params.from_address(params)), C.byref(_pointers(_lib.Inputs, fields)),
        C.byref(_pointers(_lib.Outputs, out)), C.c_void_p(scratch), scratch_bytes, _stream(device),
        C.c_void_p(event))
    return rc, list(out)


def vjp(state, forcing, geometry, cotangent, desc, vgrid, params, scratch_bytes):
    d = _lib.Desc.from_address(desc)
    device, fields = _inputs(state, forcing, geometry, d, False)
    cts = [_values(getattr(cotangent, n), d.kx * d.ix * d.il, n) for n in LEVELS]
    _on_device(device)
    cts = [t.to(device=device, dtype=torch.float32).contiguous() for t in cts]
    grads = [torch.empty(t.shape, dtype=torch.float32, device=device) for t in fields[:6]]
    grads.append(torch.empty(12, dtype=torch.float32, device=device))
    scratch = torch.empty(scratch_bytes, dtype=torch.uint8, device=device)
    rc = _lib.load().spd_vjp(
        C.byref(d), C.byref(_lib.VGrid.from_address(vgrid)),
        C.byref(_lib.Params.from_address(params)), C.byref(_pointers(_lib.Inputs, fields)),
        C.byref(_pointers(_lib.Cotangents, cts)), C.byref(_pointers(_lib.Grads, grads)),
        C.c_void_p(scratch.data_ptr()), scratch_bytes, _stream(device))
    return rc, grads


def held_suarez(state, table, out, desc):
    d = _lib.HsDesc.from_address(desc)
    columns, device = d.ix * d.il, state.temperature.device
    names = ("u_wind", "v_wind", "temperature", "normalized_surface_pressure")
    fields = [_values(getattr(state, n), columns if n == names[3] else d.kx * columns, n)
              for n in names]
    if (table.numel() != 3 * d.il or not table.is_contiguous() or table.dtype != torch.float32
            or table.device != device):
        raise ValueError("the latitude table has three values for each of the geometry's latitudes")
    for t, n in zip(out or (), LEVELS):
        _room(t, d.kx * columns, n)
    _on_device(device, out or ())
    fields = [t.to(device=device, dtype=torch.float32).contiguous() for t in fields]
    if out is None:
        out = [torch.empty_like(fields[2]) for _ in range(4)]
    p = lambda t: C.c_void_p(t.data_ptr())
    rc = _lib.load().spd_held_suarez(C.byref(d), p(table), *map(p, fields), *map(p, out),
                                     _stream(device))
    return rc, list(out)


def rollout_step(state, tendency, dt):
    """None: the caller takes torch's multi-tensor operations."""
    return None


def rollout_reverse(xbar, gradients, params, phi_sum, psa_sum, params_sum, dt):
    """None, as in rollout_step."""
    return None
