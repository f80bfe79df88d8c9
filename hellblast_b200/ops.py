"""The C ABI exposed as PyTorch custom ops (``torch.ops.hb.*``): CUDA tensors in and out, the
caller's current stream, workspace from torch's caching allocator.  Plans (geometry + lmax +
mmax + FP32 recursion checkpoints) are passed as integer ids (see geometry.py)."""
from __future__ import annotations

from typing import Optional

import torch

from . import _lib as L
from . import geometry as G


def alm_size(lmax: int, mmax: int) -> int:
    return mmax * (2 * lmax + 1 - mmax) // 2 + lmax + 1


def _prec(dtype: torch.dtype) -> int:
    if dtype in (torch.float32, torch.complex64):
        return 32
    if dtype in (torch.float64, torch.complex128):
        return 64
    raise TypeError(f"unsupported dtype {dtype}")


def _stream(dev: torch.device) -> int:
    try:
        return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device() if dev.index is None else dev.index)
    except AttributeError:  # a torch without this shortcut (2 us of host time)
        return torch.cuda.current_stream(dev).cuda_stream


def _check_cuda(*ts):
    for t in ts:
        if t is not None and not t.is_cuda:
            raise ValueError("hellblast_b200 ops take CUDA tensors (no CPU path exists)")


def _ws(p: G.Plan, prec, nmaps, dev, spin=False):
    n = p.workspace_bytes(prec, nmaps, spin)
    return torch.empty(max(n, 1), dtype=torch.uint8, device=dev)


def _wptr(w: Optional[torch.Tensor]) -> Optional[int]:
    if w is None:
        return None
    if w.dtype != torch.float64 or not w.is_contiguous():
        raise ValueError("weights must be a contiguous float64 CUDA tensor")
    return w.data_ptr()


def _ctype(prec):
    return torch.complex64 if prec == 32 else torch.complex128


def _rtype(prec):
    return torch.float32 if prec == 32 else torch.float64


_direct: dict = {}


def _op(name: str, fn):
    op = torch.library.custom_op(name, fn, mutates_args=())
    _direct[op] = fn
    return op


def _plain(args) -> bool:
    """Whether nothing but the computation can happen in a call: no tracer, mode, transform (vmap, forward AD) or
    profiler that has to see the operator, and ordinary tensors outside autograd whose storage holds their values
    (not meta or all-zero tensors, which have none, nor lazily conjugated or negated ones, which the dispatcher
    resolves on the way to the operator).  A torch that lacks one of these internal queries has no plain calls."""
    try:
        if (torch.compiler.is_compiling() or torch._C._len_torch_dispatch_stack() or torch._C._len_torch_function_stack()
                or torch._C._functorch.peek_interpreter_stack() is not None or torch._C._get_tracing_state() is not None
                or torch.autograd.forward_ad._current_level >= 0 or torch.autograd._profiler_enabled()):
            return False
    except AttributeError:
        return False
    for a in args:
        if isinstance(a, torch.Tensor) and (type(a) is not torch.Tensor or (a.requires_grad and torch.is_grad_enabled())
                                            or a.is_conj() or a.is_neg() or a.data_ptr() == 0):
            return False
    return True


def call(op, *args):
    """``op(*args)`` for one of the operators below.  Plain calls run its implementation directly:
    the custom-operator machinery takes about 11 us of host time per call, as long as the kernels of a
    whole transform at nside 16."""
    return _direct[op](*args) if _plain(args) else op(*args)


def _map2alm(maps: torch.Tensor, pid: int, weights: Optional[torch.Tensor], flags: int) -> torch.Tensor:
    _check_cuda(maps, weights)
    p = G.scalar_plan(pid, _prec(maps.dtype))
    maps = maps.contiguous()
    nmaps, prec = maps.shape[0], _prec(maps.dtype)
    out = torch.empty(nmaps, alm_size(p.lmax, p.mmax), dtype=_ctype(prec), device=maps.device)
    ws = _ws(p, prec, nmaps, maps.device)
    L.call(f"hb_map2alm_f{prec}", p.handle, nmaps, maps.data_ptr(), _wptr(weights), out.data_ptr(), ws.data_ptr(),
           ws.numel(), flags, _stream(maps.device))
    return out


map2alm = _op("hb::map2alm", _map2alm)


@map2alm.register_fake
def _(maps, pid, weights, flags):
    p = G.get_plan(pid)
    return maps.new_empty((maps.shape[0], alm_size(p.lmax, p.mmax)), dtype=_ctype(_prec(maps.dtype)))


def _alm2map(alm: torch.Tensor, pid: int, flags: int) -> torch.Tensor:
    _check_cuda(alm)
    p = G.scalar_plan(pid, _prec(alm.dtype))
    alm = alm.contiguous()
    nmaps, prec = alm.shape[0], _prec(alm.dtype)
    out = torch.empty(nmaps, p.npix, dtype=_rtype(prec), device=alm.device)
    ws = _ws(p, prec, nmaps, alm.device)
    L.call(f"hb_alm2map_f{prec}", p.handle, nmaps, alm.data_ptr(), out.data_ptr(), ws.data_ptr(), ws.numel(), flags,
           _stream(alm.device))
    return out


alm2map = _op("hb::alm2map", _alm2map)


@alm2map.register_fake
def _(alm, pid, flags):
    return alm.new_empty((alm.shape[0], G.get_plan(pid).npix), dtype=_rtype(_prec(alm.dtype)))


def _alm2map_adjoint(maps: torch.Tensor, pid: int, flags: int) -> torch.Tensor:
    _check_cuda(maps)
    p = G.scalar_plan(pid, _prec(maps.dtype))
    maps = maps.contiguous()
    nmaps, prec = maps.shape[0], _prec(maps.dtype)
    out = torch.empty(nmaps, alm_size(p.lmax, p.mmax), dtype=_ctype(prec), device=maps.device)
    ws = _ws(p, prec, nmaps, maps.device)
    L.call(f"hb_alm2map_adjoint_f{prec}", p.handle, nmaps, maps.data_ptr(), out.data_ptr(), ws.data_ptr(),
           ws.numel(), flags, _stream(maps.device))
    return out


alm2map_adjoint = _op("hb::alm2map_adjoint", _alm2map_adjoint)


@alm2map_adjoint.register_fake
def _(maps, pid, flags):
    p = G.get_plan(pid)
    return maps.new_empty((maps.shape[0], alm_size(p.lmax, p.mmax)), dtype=_ctype(_prec(maps.dtype)))


def _map2alm_adjoint(alm: torch.Tensor, pid: int, weights: Optional[torch.Tensor], flags: int) -> torch.Tensor:
    _check_cuda(alm, weights)
    p = G.scalar_plan(pid, _prec(alm.dtype))
    alm = alm.contiguous()
    nmaps, prec = alm.shape[0], _prec(alm.dtype)
    out = torch.empty(nmaps, p.npix, dtype=_rtype(prec), device=alm.device)
    ws = _ws(p, prec, nmaps, alm.device)
    L.call(f"hb_map2alm_adjoint_f{prec}", p.handle, nmaps, alm.data_ptr(), _wptr(weights), out.data_ptr(),
           ws.data_ptr(), ws.numel(), flags, _stream(alm.device))
    return out


map2alm_adjoint = _op("hb::map2alm_adjoint", _map2alm_adjoint)


@map2alm_adjoint.register_fake
def _(alm, pid, weights, flags):
    return alm.new_empty((alm.shape[0], G.get_plan(pid).npix), dtype=_rtype(_prec(alm.dtype)))


def _map2alm_spin2(Q: torch.Tensor, U: torch.Tensor, pid: int, weights: Optional[torch.Tensor],
                  flags: int) -> tuple[torch.Tensor, torch.Tensor]:
    _check_cuda(Q, U, weights)
    p = G.get_plan(pid)
    Q, U = Q.contiguous(), U.contiguous()
    nmaps, prec = Q.shape[0], _prec(Q.dtype)
    E = torch.empty(nmaps, alm_size(p.lmax, p.mmax), dtype=_ctype(prec), device=Q.device)
    B = torch.empty_like(E)
    ws = _ws(p, prec, nmaps, Q.device, spin=True)
    L.call(f"hb_map2alm_spin2_f{prec}", p.handle, nmaps, Q.data_ptr(), U.data_ptr(), _wptr(weights), E.data_ptr(),
           B.data_ptr(), ws.data_ptr(), ws.numel(), flags, _stream(Q.device))
    return E, B


map2alm_spin2 = _op("hb::map2alm_spin2", _map2alm_spin2)


@map2alm_spin2.register_fake
def _(Q, U, pid, weights, flags):
    p = G.get_plan(pid)
    e = Q.new_empty((Q.shape[0], alm_size(p.lmax, p.mmax)), dtype=_ctype(_prec(Q.dtype)))
    return e, torch.empty_like(e)


def _alm2map_spin2(E: torch.Tensor, B: torch.Tensor, pid: int, flags: int) -> tuple[torch.Tensor, torch.Tensor]:
    _check_cuda(E, B)
    p = G.get_plan(pid)
    E, B = E.contiguous(), B.contiguous()
    nmaps, prec = E.shape[0], _prec(E.dtype)
    Q = torch.empty(nmaps, p.npix, dtype=_rtype(prec), device=E.device)
    U = torch.empty_like(Q)
    ws = _ws(p, prec, nmaps, E.device, spin=True)
    L.call(f"hb_alm2map_spin2_f{prec}", p.handle, nmaps, E.data_ptr(), B.data_ptr(), Q.data_ptr(), U.data_ptr(),
           ws.data_ptr(), ws.numel(), flags, _stream(E.device))
    return Q, U


alm2map_spin2 = _op("hb::alm2map_spin2", _alm2map_spin2)


@alm2map_spin2.register_fake
def _(E, B, pid, flags):
    q = E.new_empty((E.shape[0], G.get_plan(pid).npix), dtype=_rtype(_prec(E.dtype)))
    return q, torch.empty_like(q)


def _alm2map_spin2_adjoint(gQ: torch.Tensor, gU: torch.Tensor, pid: int,
                          flags: int) -> tuple[torch.Tensor, torch.Tensor]:
    _check_cuda(gQ, gU)
    p = G.get_plan(pid)
    gQ, gU = gQ.contiguous(), gU.contiguous()
    nmaps, prec = gQ.shape[0], _prec(gQ.dtype)
    gE = torch.empty(nmaps, alm_size(p.lmax, p.mmax), dtype=_ctype(prec), device=gQ.device)
    gB = torch.empty_like(gE)
    ws = _ws(p, prec, nmaps, gQ.device, spin=True)
    L.call(f"hb_alm2map_spin2_adjoint_f{prec}", p.handle, nmaps, gQ.data_ptr(), gU.data_ptr(), gE.data_ptr(),
           gB.data_ptr(), ws.data_ptr(), ws.numel(), flags, _stream(gQ.device))
    return gE, gB


alm2map_spin2_adjoint = _op("hb::alm2map_spin2_adjoint", _alm2map_spin2_adjoint)


@alm2map_spin2_adjoint.register_fake
def _(gQ, gU, pid, flags):
    p = G.get_plan(pid)
    e = gQ.new_empty((gQ.shape[0], alm_size(p.lmax, p.mmax)), dtype=_ctype(_prec(gQ.dtype)))
    return e, torch.empty_like(e)


def _map2alm_spin2_adjoint(gE: torch.Tensor, gB: torch.Tensor, pid: int, weights: Optional[torch.Tensor],
                          flags: int) -> tuple[torch.Tensor, torch.Tensor]:
    _check_cuda(gE, gB, weights)
    p = G.get_plan(pid)
    gE, gB = gE.contiguous(), gB.contiguous()
    nmaps, prec = gE.shape[0], _prec(gE.dtype)
    gQ = torch.empty(nmaps, p.npix, dtype=_rtype(prec), device=gE.device)
    gU = torch.empty_like(gQ)
    ws = _ws(p, prec, nmaps, gE.device, spin=True)
    L.call(f"hb_map2alm_spin2_adjoint_f{prec}", p.handle, nmaps, gE.data_ptr(), gB.data_ptr(), _wptr(weights),
           gQ.data_ptr(), gU.data_ptr(), ws.data_ptr(), ws.numel(), flags, _stream(gE.device))
    return gQ, gU


map2alm_spin2_adjoint = _op("hb::map2alm_spin2_adjoint", _map2alm_spin2_adjoint)


@map2alm_spin2_adjoint.register_fake
def _(gE, gB, pid, weights, flags):
    q = gE.new_empty((gE.shape[0], G.get_plan(pid).npix), dtype=_rtype(_prec(gE.dtype)))
    return q, torch.empty_like(q)


def _alm2cl(alm1: torch.Tensor, alm2: Optional[torch.Tensor], lmax: int, mmax: int) -> torch.Tensor:
    _check_cuda(alm1, alm2)
    alm1 = alm1.contiguous()
    if alm2 is not None:
        alm2 = alm2.contiguous().to(alm1.dtype)
    nmaps, prec = alm1.shape[0], _prec(alm1.dtype)
    cl = torch.empty(nmaps, lmax + 1, dtype=torch.float64, device=alm1.device)
    L.call(f"hb_alm2cl_f{prec}", lmax, mmax, nmaps, alm1.data_ptr(), None if alm2 is None else alm2.data_ptr(),
           cl.data_ptr(), _stream(alm1.device))
    return cl


alm2cl = _op("hb::alm2cl", _alm2cl)


@alm2cl.register_fake
def _(alm1, alm2, lmax, mmax):
    return alm1.new_empty((alm1.shape[0], lmax + 1), dtype=torch.float64)


def ring_tables(nside: int, phi0_mode: int, device) -> dict:
    """Device ring tables from the hb_ring_tables kernel."""
    nr = 4 * nside - 1
    dev = torch.device(device)
    f64 = dict(dtype=torch.float64, device=dev)
    out = dict(z=torch.empty(nr, **f64), theta=torch.empty(nr, **f64),
               nphi=torch.empty(nr, dtype=torch.int32, device=dev), phi0=torch.empty(nr, **f64),
               ring_start=torch.empty(nr + 1, dtype=torch.int64, device=dev), z_edges=torch.empty(nr + 1, **f64),
               weights_dz=torch.empty(nr, **f64))
    L.call("hb_ring_tables", nside, phi0_mode, out["z"].data_ptr(), out["theta"].data_ptr(), out["nphi"].data_ptr(),
           out["phi0"].data_ptr(), out["ring_start"].data_ptr(), out["z_edges"].data_ptr(),
           out["weights_dz"].data_ptr(), _stream(dev))
    return out
