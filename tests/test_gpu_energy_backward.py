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
