"""Variational energy Re<psi|H|psi> / <psi|psi> with FP64 reductions.

The reference evaluates this on the caller side (qmb/vmc.py:104-116,
qmb/haar.py:491) with the Hamiltonian application detached from autograd.
Here the energy backpropagates into psi (and from there into whatever
produced psi).  For a Hermitian operator (checked once per compiled table)
the gradient needs H psi only: dE/dpsi* = (H psi - E psi) / <psi|psi>, so one
term walk serves the energy and its gradient.  Otherwise H psi goes through
``Hamiltonian.apply_within``'s autograd function, whose backward is the
adjoint kernel.  complex64 amplitudes use the compensated FP32 kernels; the
diagonal term, the norm and the quotient stay in FP64.
"""

from __future__ import annotations

import torch

from . import _native
from .hamiltonian import Hamiltonian, _plain

__all__ = ["variational_energy"]


class _HermitianEnergy(torch.autograd.Function):
    """E = Re<psi|H psi> / <psi|psi> for Hermitian H; backward from the saved H psi."""

    @staticmethod
    def forward(ctx, ham: Hamiltonian, configs, psi):
        given, psi = psi, _plain(psi.detach())
        if psi.dtype == torch.complex64:
            hpsi = ham.apply_within_compensated(configs, psi, configs)
        else:
            hpsi = ham.apply_within(configs, psi, configs)
        sums = torch.empty(2, dtype=torch.float64, device=psi.device)
        with torch.cuda.device(psi.device):
            scratch = torch.empty(1024, dtype=torch.float64, device=psi.device)
            _native.call("qmbx_energy", psi.shape[0], int(psi.dtype == torch.complex64), psi.data_ptr(), hpsi.data_ptr(),
                         sums.data_ptr(), scratch.data_ptr(), torch.cuda.current_stream(psi.device).cuda_stream)
        if psi.dtype == torch.complex64 and psi.data_ptr() == given.data_ptr():
            psi = psi.clone()  # a caller may change complex64 amplitudes in place before the backward
        ctx.save_for_backward(hpsi, psi, sums)
        return sums[0].clone()

    @staticmethod
    def backward(ctx, grad):
        hpsi, psi, sums = ctx.saved_tensors
        # torch's gradient of a real loss in a complex input is 2 dL/dpsi*
        composed = torch.is_grad_enabled()  # a graph of the gradient was asked for: it is linear in grad
        if not composed:
            grad = grad.to(torch.float64).contiguous()
            try:
                grad_ptr = grad.data_ptr()
            except RuntimeError:  # a batch of gradients (is_grads_batched) has no memory of its own
                composed = True
        if composed:
            g = grad * 2.0 * (hpsi - sums[0] * psi.to(torch.complex128)) / sums[1]
            return None, None, g.to(psi.dtype)
        g = torch.empty_like(psi)
        with torch.cuda.device(psi.device):
            _native.call("qmbx_energy_grad", psi.shape[0], int(psi.dtype == torch.complex64), psi.data_ptr(),
                         hpsi.data_ptr(), sums.data_ptr(), grad_ptr, g.data_ptr(),
                         torch.cuda.current_stream(psi.device).cuda_stream)
        return None, None, g


def variational_energy(ham: Hamiltonian, configs: torch.Tensor, psi: torch.Tensor, *,
                       hermitian_shortcut: bool = True) -> torch.Tensor:
    """Re<psi|H|psi> / <psi|psi> over one set of configurations; a float64 scalar.

    With ``hermitian_shortcut`` (the default) a Hermitian operator takes its
    gradient from the saved H psi; ``hermitian_shortcut=False`` always sends
    the backward pass through the adjoint kernel (``apply_within``'s autograd
    function), which the gradient checks use to exercise that kernel.
    """
    if psi.dtype not in (torch.complex64, torch.complex128):
        raise RuntimeError("psi must be complex64 or complex128")
    if hermitian_shortcut and psi.requires_grad and torch.is_grad_enabled() and configs.dim() == 2 and \
            ham._table(configs.device, configs.shape[1]).hermitian:
        return _HermitianEnergy.apply(ham, configs, psi)
    if psi.dtype == torch.complex64:
        hpsi = ham.apply_within_compensated(configs, psi, configs)
    elif psi.dtype == torch.complex128:
        hpsi = ham.apply_within(configs, psi, configs)
    else:
        raise RuntimeError("psi must be complex64 or complex128")
    psi64 = psi.to(torch.complex128)
    numerator = torch.sum(psi64.conj() * hpsi).real
    denominator = torch.sum(psi64.conj() * psi64).real
    return numerator / denominator
