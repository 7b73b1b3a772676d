"""Scan or walk, as the device chooses from a sample of the rows.

A set that holds all or most neighbours of its rows is walked, a thin or
clustered one of many terms scanned; forwards, both backwards, the adjoint and
the matrix give what the grouped walk gives either way (sums of fewer than
14,000 products in another order).
"""

from __future__ import annotations

import pytest
import torch

from qmb_gb300 import Hamiltonian, terms
from test_gpu_pair_list import TOL, _magnitudes, _psi, _scanned

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("orbits,alpha,beta,n,scanned", [
    (14, 2, 2, 0, False),       # every determinant: 8,281 rows, 756 neighbours each
    (12, 4, 4, 0, False),       # 245,025 rows, 1,424 neighbours each
    (14, 5, 5, 30000, True),    # 30,000 of 4.0M rows
    (20, 5, 5, 20000, True),
])
def test_choice(orbits, alpha, beta, n, scanned, cuda_device, monkeypatch):
    monkeypatch.delenv("QMBX_WALK", raising=False)
    table = terms.integral_hamiltonian_tables(orbits, seed=101)
    ham, bound = Hamiltonian(table, kind="fermi"), _magnitudes(table)
    rows = torch.from_numpy(terms.random_determinants(orbits, alpha, beta, n, seed=102) if n else
                            terms.all_determinants(orbits, alpha, beta)).to(cuda_device)
    for c_i, c_j in ((rows, rows), (rows[::2].contiguous(), rows)):
        psi, g = _psi(c_i.shape[0], 103, cuda_device), _psi(c_j.shape[0], 104, cuda_device)
        assert _scanned(ham._table(cuda_device, rows.shape[1]), c_i, c_j, psi, cuda_device) == scanned
        got = []
        for first_guess in (1 << 22, 16):
            fresh = Hamiltonian(table, kind="fermi")
            fresh._LOG_FIRST_GUESS = first_guess
            p = psi.clone().requires_grad_(True)
            y = fresh.apply_within(c_i, p, c_j)
            got.append((y.detach(), torch.autograd.grad(y, p, grad_outputs=g)[0]))
        adjoint = ham.apply_within_adjoint(c_i, g, c_j)
        with monkeypatch.context() as walked:
            walked.setenv("QMBX_WALK", "grouped")
            want, want_back = ham.apply_within(c_i, psi, c_j), ham.apply_within_adjoint(c_i, g, c_j)
            size = bound.apply_within(c_i, psi.abs().to(torch.complex128), c_j).abs()
            size_back = bound.apply_within_adjoint(c_i, g.abs().to(torch.complex128), c_j).abs()
        for y, back in got:
            assert torch.all((y - want).abs() <= TOL * size)
            assert torch.all((back - want_back).abs() <= TOL * size_back)
        assert torch.all((adjoint - want_back).abs() <= TOL * size_back)
    x = _psi(rows.shape[0], 105, cuda_device)
    mat = ham.matrix(rows)
    with monkeypatch.context() as walked:
        walked.setenv("QMBX_WALK", "grouped")
        other = ham.matrix(rows)
        size = bound.apply_within(rows, x.abs().to(torch.complex128), rows).abs()
    assert torch.equal(mat.row_ptr, other.row_ptr)
    assert torch.all((mat.apply(x) - other.apply(x)).abs() <= TOL * size)


@pytest.mark.parametrize("first,then", [(None, "scan"), ("scan", None), ("scan", "grouped"), ("grouped", "scan")])
@pytest.mark.parametrize("first_guess", [1 << 20, 16])
def test_environment_changed_before_the_backward(first, then, first_guess, cuda_device, monkeypatch):
    table = terms.integral_hamiltonian_tables(9, seed=106, complex_valued=True)
    ham = Hamiltonian(table, kind="fermi")
    ham._LOG_FIRST_GUESS = first_guess
    rows = torch.from_numpy(terms.random_determinants(9, 4, 4, 900, seed=107)).to(cuda_device)
    psi, g = _psi(900, 108, cuda_device).requires_grad_(True), _psi(900, 109, cuda_device)
    set_to = lambda walk: monkeypatch.setenv("QMBX_WALK", walk) if walk else monkeypatch.delenv("QMBX_WALK", raising=False)
    set_to(first)
    y = ham.apply_within(rows, psi, rows)
    set_to(then)
    (back,) = torch.autograd.grad(y, psi, grad_outputs=g)
    set_to("grouped")
    want = ham.apply_within_adjoint(rows, g, rows)
    size = _magnitudes(table).apply_within_adjoint(rows, g.abs().to(torch.complex128), rows).abs()
    assert torch.all((back - want).abs() <= TOL * size)
