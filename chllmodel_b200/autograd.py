"""``torch.autograd.Function`` over the hand-written energy adjoint kernel.

``lattice_energy(n, s, eps, K, h, shape, boundary)`` returns the FP64 total
energy of a lattice whose directors ``n`` (N x 3, FP32, CUDA, natural order
i fastest) and chiralities ``s`` (N, +-1) are torch tensors; its backward
pass comes from the adjoint kernel (``natural_grad_kernel``, on the tensors as
they are: dE/dn for every site, plus dE/deps, dE/dK, dE/dh in FP64), not from
autograd tracing.  The Metropolis sweep itself is not differentiated:
acceptance stays exactly the reference's rule (chll_mod.f90:188-200).

``quench`` runs the zero-temperature gradient descent on the device, and
``coupling_sensitivities`` returns dE/d(eps, K, h) of a lattice state.
This module is the only place the package uses torch on the compute side.
"""
from __future__ import annotations

import ctypes as ct

import torch

from . import _lib
from ._lib import Coupling
from .lattice import Lattice, coupling


def _natural(n, s, eps, K, h, shape, boundary, project, want_grad, energy, derivs):
    """The adjoint of CUDA tensors n (N, 3) and s (N,) on n's device, enqueued
    on its current stream: E into energy, dE/d(eps, K, h) into derivs (FP64),
    and the gradient (N, 3), FP32, returned if wanted."""
    ni, nj, nk = (int(x) for x in shape)
    if boundary not in ("open", "periodic"):
        raise ValueError("boundary must be 'open' or 'periodic'")
    if s.device != n.device:
        raise RuntimeError(f"n and s must be on one device (got {n.device} and {s.device})")
    n32 = n.detach().to(torch.float32).contiguous()
    s32 = s.detach().to(torch.float32).contiguous()
    grad = torch.empty_like(n32) if want_grad else None
    work = torch.empty(_lib.GRAD_WORK, dtype=torch.float64, device=n.device)
    cp = Coupling(0.0, float(K), float(h), float(eps))
    with torch.cuda.device(n.device):
        _lib.check(_lib.load().chll_energy_grad_natural(
            n32.data_ptr(), s32.data_ptr(), ni, nj, nk,
            _lib.CHLL_PERIODIC if boundary == "periodic" else _lib.CHLL_OPEN, ct.byref(cp),
            int(bool(project)), grad.data_ptr() if want_grad else None, energy.data_ptr(),
            derivs.data_ptr(), work.data_ptr(), torch.cuda.current_stream().cuda_stream))
    return grad


class LatticeEnergy(torch.autograd.Function):
    @staticmethod
    def forward(ctx, n, s, eps, K, h, shape, boundary):
        if not n.is_cuda:
            raise ValueError("lattice_energy needs CUDA tensors (the kernels have no CPU path)")
        N = int(shape[0]) * int(shape[1]) * int(shape[2])
        if n.shape != (N, 3) or s.numel() != N:
            raise ValueError(f"n must be ({N}, 3) and s ({N},) for lattice {tuple(shape)}")
        energy = torch.empty((), dtype=torch.float64, device=n.device)
        derivs = torch.empty(3, dtype=torch.float64, device=n.device)
        grad = _natural(n, s, eps, K, h, shape, boundary, False, ctx.needs_input_grad[0], energy,
                        derivs)
        ctx.on_host = not (eps.is_cuda or K.is_cuda or h.is_cuda)
        ctx.save_for_backward(grad.to(n.dtype) if grad is not None else None, derivs)
        return energy

    @staticmethod
    def backward(ctx, g_out):
        grad_n, d_couplings = ctx.saved_tensors
        g = g_out.to(torch.float64)
        gn = (g * grad_n) if ctx.needs_input_grad[0] else None
        ge = gk = gh = None
        if any(ctx.needs_input_grad[2:5]):
            gc = g * d_couplings
            if ctx.on_host:
                gc = gc.cpu()  # one copy for the three
            ge, gk, gh = (v if need else None
                          for v, need in zip(gc.unbind(), ctx.needs_input_grad[2:5]))
        return gn, None, ge, gk, gh, None, None


def lattice_energy(n, s, eps, K, h, shape, boundary="periodic"):
    """Total energy (FP64) with analytic gradients to n, eps, K and h.

    eps, K, h may be python floats or 0-d tensors (requires_grad for their
    derivatives)."""
    as_t = lambda v: v if torch.is_tensor(v) else torch.tensor(float(v), dtype=torch.float64)
    return LatticeEnergy.apply(n, s, as_t(eps), as_t(K), as_t(h), tuple(shape), boundary)


def _on_gpu(n: torch.Tensor, s: torch.Tensor, shape):
    """n and s checked against the lattice, on a GPU (host tensors are copied)."""
    N = int(shape[0]) * int(shape[1]) * int(shape[2])
    if n.ndim != 2 or n.shape[1] != 3 or n.shape[0] < N or s.numel() != n.shape[0]:
        raise ValueError(f"n must be ({N}, 3) and s ({N},) for lattice {tuple(shape)}")
    if not n.is_cuda and not s.is_cuda:
        return n.to("cuda:0"), s.to("cuda:0")
    return n, s


def tangent_gradient(n, s, eps, K, h, shape, boundary="periodic") -> torch.Tensor:
    """(I - n n^T) dE/dn: the torque direction on every director."""
    gn, gs = _on_gpu(n, s, shape)
    out = torch.empty(4, dtype=torch.float64, device=gn.device)
    return _natural(gn, gs, eps, K, h, shape, boundary, True, True, out, out[1:]).to(n.device)


def coupling_sensitivities(n, s, eps, K, h, shape, boundary="periodic") -> dict:
    """E and dE/d(eps, K, h) of a lattice state, FP64."""
    gn, gs = _on_gpu(n, s, shape)
    out = torch.empty(4, dtype=torch.float64, device=gn.device)
    _natural(gn, gs, eps, K, h, shape, boundary, False, False, out, out[1:])
    E, de, dk, dh = out.cpu().numpy()
    return {"E": E, "dE_deps": de, "dE_dK": dk, "dE_dh": dh}


def quench(lat: Lattice, eps: float, K: float, h: float, eta: float, nsteps: int,
           report_every: int = 0):
    """Zero-temperature gradient quench of a device lattice: nsteps of
    n <- normalise(n - eta (I - n n^T) dE/dn), colour by colour.  Returns the
    FP64 energies after every `report_every` steps (and at the end)."""
    cp = coupling(0.0, K, h, eps)
    energies = []
    done = 0
    chunk = report_every if report_every > 0 else nsteps
    while done < nsteps:
        step = min(chunk, nsteps - done)
        lat.quench(cp, eta, step)
        done += step
        energies.append((done, lat.energy_sums(cp)[0]))
    return energies
