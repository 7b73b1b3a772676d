"""Grouped walks that share a row among the warps of a block, at the team sizes' edges, against the oracle.

Both precisions, forward and backward (gathers and scatters), rows that do not
fill the last block, and a repeated call that gives the same bits.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle
from qmb_gb300 import Hamiltonian, terms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_i,n_j", [(1, 0), (9, 500), (1215, 0), (1216, 0), (2431, 0), (2433, 0), (4863, 0), (4864, 0), (1300, 4000)])
def test_teams_match_the_oracle(n_i, n_j, cuda_device, monkeypatch):
    monkeypatch.setenv("QMBX_WALK", "grouped")
    n = 8
    site, kind, coef = (x.numpy() for x in terms.integral_hamiltonian_tables(n, seed=71, complex_valued=True))
    ci = terms.random_determinants(n, 4, 4, n_i, seed=72)
    cj = terms.random_determinants(n, 4, 4, n_j, seed=73) if n_j else ci
    ham = Hamiltonian((torch.from_numpy(site), torch.from_numpy(kind), torch.from_numpy(coef)), kind="fermi")
    di = torch.from_numpy(ci).to(cuda_device)
    dj = torch.from_numpy(cj).to(cuda_device) if n_j else di
    psi, gj = terms.random_psi(ci.shape[0], seed=74), terms.random_psi(cj.shape[0], seed=75)
    scale = np.abs(coef).sum() * max(np.abs(psi).max(), np.abs(gj).max())
    for dtype, tol in ((np.complex128, 1e-13), (np.complex64, 2e-7)):
        p = torch.from_numpy(psi.astype(dtype)).to(cuda_device).requires_grad_(True)
        y = ham.apply_within(di, p, dj)
        (back,) = torch.autograd.grad(y, p, grad_outputs=torch.from_numpy(gj.astype(dtype)).to(cuda_device))
        want = oracle.apply_within(site, kind, coef, ci, psi.astype(dtype).astype(np.complex128), cj, 1)
        assert np.all(np.abs(y.detach().cpu().numpy() - want) <= tol * scale)
        want = oracle.apply_within_adjoint(site, kind, coef, ci, cj, gj.astype(dtype).astype(np.complex128), 1)
        assert np.all(np.abs(back.cpu().numpy() - want) <= tol * scale)
    monkeypatch.setenv("QMBX_DETERMINISTIC", "1")
    one, two = (ham.apply_within(di, torch.from_numpy(psi).to(cuda_device), dj) for _ in range(2))
    assert torch.equal(one, two)
