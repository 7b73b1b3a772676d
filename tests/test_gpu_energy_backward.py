"""What variational_energy's backward accepts: amplitudes changed in place meanwhile, batches of gradients.

The same gradient formed with torch operations from the same H psi differs by
a few FP64 roundings, or one FP32 rounding of the result.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from qmb_gb300 import Hamiltonian, terms, variational_energy

pytestmark = pytest.mark.gpu


def _system(device, dtype, n=700):
    site, kind, coef = terms.integral_hamiltonian_tables(8, seed=85)
    rows = torch.from_numpy(terms.random_determinants(8, 4, 4, n, seed=86)).to(device)
    psi = torch.from_numpy(terms.random_psi(n, seed=87)).to(device).to(dtype)
    return Hamiltonian((site, kind, coef), kind="fermi"), rows, psi


def test_complex64_changed_in_place(cuda_device):
    ham, rows, psi = _system(cuda_device, torch.complex64)
    (want,) = torch.autograd.grad(variational_energy(ham, rows, psi.requires_grad_(True)), psi)
    energy = variational_energy(ham, rows, psi)
    with torch.no_grad():
        psi.mul_(0.5)
    (got,) = torch.autograd.grad(energy, psi)
    assert (got - want).abs().max().item() <= 1e-6 * want.abs().max().item()


@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64])
def test_batched_gradients(dtype, cuda_device):
    ham, rows, psi = _system(cuda_device, dtype)
    energy = variational_energy(ham, rows, psi.requires_grad_(True))
    weights = torch.tensor([1.0, -2.0, 0.25], dtype=torch.float64, device=cuda_device)
    (got,) = torch.autograd.grad(energy, psi, grad_outputs=weights, is_grads_batched=True, retain_graph=True)
    tol = 1e-13 if dtype == torch.complex128 else 1e-6
    for k in range(3):
        (want,) = torch.autograd.grad(energy, psi, grad_outputs=weights[k], retain_graph=True)
        assert (got[k] - want).abs().max().item() <= tol * want.abs().max().item()
