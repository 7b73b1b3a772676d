"""Tiled walks that leave out terms no looked-up row can be reached by (rows of two key words or more).

Rows of which none, some and nearly all share a word with others, one set and
two, both precisions, forward and backward, against the oracle.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle
from qmb_gb300 import Hamiltonian, terms

pytestmark = pytest.mark.gpu

N = 65536 + 77  # just above the line


def _rows(n_qubytes, sites, shift, kind, seed):
    rng = np.random.default_rng(seed)
    if kind == "random":
        bits = rng.random((N + 64, sites)) < 0.5
    elif kind == "halves":  # few left halves, few right ones
        left = rng.random((300, sites // 2)) < 0.5
        right = rng.random((300, sites - sites // 2)) < 0.5
        pick = rng.permutation(300 * 300)[:N + 64]
        bits = np.concatenate([left[pick // 300], right[pick % 300]], axis=1)
    else:  # chains of hops from random rows
        base = rng.random((N // 4, sites)) < 0.5
        bits = np.repeat(base, 8, axis=0)
        for k in range(1, 8):
            at = rng.integers(0, sites - 2, size=base.shape[0])
            r = np.arange(base.shape[0]) * 8 + k
            bits[r, at], bits[r, at + 2] = bits[r, at + 2].copy(), bits[r, at].copy()
    wide = np.zeros((bits.shape[0], 8 * n_qubytes), dtype=np.uint8)
    wide[:, shift:shift + sites] = bits
    return terms.unique_rows(terms.pack_sites(wide, n_qubytes))[:N]


@pytest.mark.parametrize("n_qubytes,shift", [(10, 4), (17, 40)])
@pytest.mark.parametrize("kinds", [("random", None), ("halves", None), ("chains", None), ("chains", "halves"), ("halves", "chains")])
def test_reach_matches_the_oracle(n_qubytes, shift, kinds, cuda_device):
    site, kind, coef = (x.numpy() for x in terms.sort_terms(*terms.prepare(terms.hubbard_dict(6, 6, 1.0, 4.0))))
    site = np.where(kind == 2, site, site + shift).astype(np.int16)
    ci = _rows(n_qubytes, 72, shift, kinds[0], 51)
    cj = ci if kinds[1] is None else _rows(n_qubytes, 72, shift, kinds[1], 52)
    if kinds[1] is not None:
        cj = terms.unique_rows(np.concatenate([cj, ci[N // 2:]]))
    assert min(ci.shape[0], cj.shape[0]) >= 65536
    ham = Hamiltonian((torch.from_numpy(site), torch.from_numpy(kind), torch.from_numpy(coef)), kind="fermi")
    di = torch.from_numpy(ci).to(cuda_device)
    dj = di if cj is ci else torch.from_numpy(cj).to(cuda_device)
    psi, gj = terms.random_psi(ci.shape[0], seed=53), terms.random_psi(cj.shape[0], seed=54)
    scale = np.abs(coef).sum() * max(np.abs(psi).max(), np.abs(gj).max())
    for dtype, tol in ((np.complex128, 1e-12), (np.complex64, 2e-7)):
        p = torch.from_numpy(psi.astype(dtype)).to(cuda_device).requires_grad_(True)
        y = ham.apply_within(di, p, dj)
        (back,) = torch.autograd.grad(y, p, grad_outputs=torch.from_numpy(gj.astype(dtype)).to(cuda_device))
        want = oracle.apply_within(site, kind, coef, ci, psi.astype(dtype).astype(np.complex128), cj, 1)
        assert np.all(np.abs(y.detach().cpu().numpy() - want) <= tol * scale)
        want = oracle.apply_within_adjoint(site, kind, coef, ci, cj, gj.astype(dtype).astype(np.complex128), 1)
        assert np.all(np.abs(back.cpu().numpy() - want) <= tol * scale)


@pytest.mark.parametrize("kind", ["random", "halves", "chains"])
@pytest.mark.parametrize("more", [0, 500])
def test_reach_with_the_rows_copied(kind, more, cuda_device):
    # the looked-up set holds a copy of every walked row, and `more` others
    site, kinds, coef = (x.numpy() for x in terms.sort_terms(*terms.prepare(terms.hubbard_dict(6, 6, 1.0, 4.0))))
    shift, n_qubytes = 4, 10
    site = np.where(kinds == 2, site, site + shift).astype(np.int16)
    ci = _rows(n_qubytes, 72, shift, kind, 61)
    cj = ci if more == 0 else terms.unique_rows(np.concatenate([ci, _rows(n_qubytes, 72, shift, "random", 62)[:more]]))
    ham = Hamiltonian((torch.from_numpy(site), torch.from_numpy(kinds), torch.from_numpy(coef)), kind="fermi")
    di, dj = torch.from_numpy(ci).to(cuda_device), torch.from_numpy(cj.copy()).to(cuda_device)
    psi, gj = terms.random_psi(ci.shape[0], seed=63), terms.random_psi(cj.shape[0], seed=64)
    scale = np.abs(coef).sum() * max(np.abs(psi).max(), np.abs(gj).max())
    for dtype, tol in ((np.complex128, 1e-12), (np.complex64, 2e-7)):
        p = torch.from_numpy(psi.astype(dtype)).to(cuda_device).requires_grad_(True)
        y = ham.apply_within(di, p, dj)
        (back,) = torch.autograd.grad(y, p, grad_outputs=torch.from_numpy(gj.astype(dtype)).to(cuda_device))
        want = oracle.apply_within(site, kinds, coef, ci, psi.astype(dtype).astype(np.complex128), cj, 1)
        assert np.all(np.abs(y.detach().cpu().numpy() - want) <= tol * scale)
        want = oracle.apply_within_adjoint(site, kinds, coef, ci, cj, gj.astype(dtype).astype(np.complex128), 1)
        assert np.all(np.abs(back.cpu().numpy() - want) <= tol * scale)
