"""Amplitudes whose conjugation or sign torch only marks give what their values give, bit for bit."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from qmb_gb300 import Hamiltonian, terms, variational_energy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64])
@pytest.mark.parametrize("lazy", [torch.conj, torch._neg_view])
def test_lazy_amplitudes(dtype, lazy, cuda_device):
    table = terms.integral_hamiltonian_tables(8, seed=131, complex_valued=True)
    ham = Hamiltonian(table, kind="fermi")
    rows = torch.from_numpy(terms.random_determinants(8, 4, 4, 600, seed=132)).to(cuda_device)
    psi = torch.from_numpy(terms.random_psi(600, seed=133)).to(cuda_device).to(dtype)
    marked, plain = lazy(psi), lazy(psi).resolve_conj().resolve_neg().clone()
    assert marked.is_conj() or marked.is_neg()
    assert torch.equal(ham.apply_within(rows, marked, rows), ham.apply_within(rows, plain, rows))
    assert torch.equal(ham.apply_within_adjoint(rows, marked, rows), ham.apply_within_adjoint(rows, plain, rows))
    assert torch.equal(ham.find_relative(rows, marked, 50), ham.find_relative(rows, plain, 50))
    assert ham.pt2(rows, marked, 50) == pytest.approx(ham.pt2(rows, plain, 50), rel=1e-12)
    assert variational_energy(ham, rows, marked).item() == pytest.approx(variational_energy(ham, rows, plain).item(), rel=1e-12)
    if dtype == torch.complex128:
        mat = ham.matrix(rows)
        assert torch.equal(mat.apply(marked), mat.apply(plain))
    # gradients that arrive marked
    p = psi.clone().requires_grad_(True)
    (got,) = torch.autograd.grad(ham.apply_within(rows, p, rows), p, grad_outputs=marked)
    (want,) = torch.autograd.grad(ham.apply_within(rows, p, rows), p, grad_outputs=plain)
    assert (got - want).abs().max().item() <= (1e-13 if dtype == torch.complex128 else 1e-6) * want.abs().max().item()
