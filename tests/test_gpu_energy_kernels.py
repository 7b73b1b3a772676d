"""The energy and gradient kernels against numpy in FP64, at block edges and in both precisions.

FP64 to n 2^-52 of the sums of magnitudes; the FP32 gradient to its rounding.
The gradient of the gradient stays linear in the incoming one.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle
from qmb_gb300 import Hamiltonian, terms, variational_energy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 257, 4800])
@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
def test_energy_and_gradient(n, dtype, cuda_device):
    site, kind, coef = (x.numpy() for x in terms.integral_hamiltonian_tables(8, seed=81, complex_valued=False))
    rows = terms.random_determinants(8, 4, 4, n, seed=82)
    psi = terms.random_psi(n, seed=83).astype(dtype)
    ham = Hamiltonian((torch.from_numpy(site), torch.from_numpy(kind), torch.from_numpy(coef)), kind="fermi")
    c = torch.from_numpy(rows).to(cuda_device)
    p = torch.from_numpy(psi).to(cuda_device).requires_grad_(True)
    energy = variational_energy(ham, c, p)
    (grad,) = torch.autograd.grad(3.0 * energy, p)
    p64 = psi.astype(np.complex128)
    h = oracle.apply_within(site, kind, coef, rows, p64, rows)
    norm = np.vdot(p64, p64).real
    want = np.vdot(p64, h).real / norm
    size = np.abs(coef).sum()
    assert abs(energy.item() - want) <= (n * 2.0**-52 + 1e-13) * size
    want_grad = 6.0 * (h - want * p64) / norm
    tol = 1e-12 if dtype == np.complex128 else 2e-7
    assert np.all(np.abs(grad.cpu().numpy() - want_grad) <= tol * 6.0 * size * np.abs(p64).max() / norm)
    again = variational_energy(ham, c, p)
    weight = torch.tensor(2.0, dtype=torch.float64, device=cuda_device, requires_grad=True)
    (first,) = torch.autograd.grad(again, p, grad_outputs=weight, create_graph=True)
    (slope,) = torch.autograd.grad(first.real.sum() + first.imag.sum(), weight)
    want_slope = (want_grad / 3.0).real.sum() + (want_grad / 3.0).imag.sum()
    assert abs(slope.item() - want_slope) <= 1e-6 * np.abs(want_grad).sum() + 1e-12
