"""Diagonal passes by the rows' own groups against the oracle, on tables above the tiled line.

Rows of no, one, odd, many and all particles (the lanes' shares of positions),
row counts around a block's 32, one to four key words, terms of occupations
only and terms that also test empty sites or more than two sites.  FP64 to
1e-12 of the absolute sum, the compensated FP32 path to 2e-7.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle
from qmb_gb300 import Hamiltonian, terms

pytestmark = pytest.mark.gpu


def _table(sites, conditioned):
    rng = np.random.default_rng(41)
    out = {(): 0.7}
    for a in range(sites):
        out[((a, 1), (a, 0))] = complex(*rng.standard_normal(2))
        for b in range(a):
            out[((a, 1), (a, 0), (b, 1), (b, 0))] = complex(rng.standard_normal(), 0.0)
            if conditioned and (a + b) % 3 == 0:
                out[((a, 1), (a, 0), (b, 0), (b, 1))] = complex(*rng.standard_normal(2))  # b empty
    out[((0, 1), (1, 0))] = out[((1, 1), (0, 0))] = 0.5
    return tuple(x.numpy() for x in terms.sort_terms(*terms.prepare(out)))


@pytest.mark.parametrize("n_qubytes", [3, 8, 11, 20, 32])
@pytest.mark.parametrize("conditioned", [False, True])
@pytest.mark.parametrize("n", [1, 31, 33, 700])
def test_diagonal_matches_the_oracle(n_qubytes, conditioned, n, cuda_device):
    sites = min(8 * n_qubytes, 40)
    site, kind, coef = _table(sites, conditioned)
    site = np.where(kind == 2, site, site + 8 * n_qubytes - sites).astype(np.int16)
    rng = np.random.default_rng(42)
    bits = np.zeros((n, 8 * n_qubytes), dtype=np.uint8)
    fill = rng.integers(0, sites + 1, size=n)
    fill[0] = sites
    if n > 2:
        fill[1], fill[2] = 0, 1
    for r in range(n):
        bits[r, 8 * n_qubytes - sites + rng.permutation(sites)[:fill[r]]] = 1
    rows = terms.unique_rows(terms.pack_sites(bits, n_qubytes))
    ham = Hamiltonian((torch.from_numpy(site), torch.from_numpy(kind), torch.from_numpy(coef)), kind="fermi")
    dev = torch.from_numpy(rows).to(cuda_device)
    got = ham.diagonal_term(dev).cpu().numpy()
    want = oracle.diagonal_term(site, kind, coef, rows)
    total = np.abs(coef).sum()
    assert np.all(np.abs(got - want) <= 1e-12 * total)
    psi = terms.random_psi(rows.shape[0], seed=43)
    for dtype, tol in ((np.complex128, 1e-12), (np.complex64, 2e-7)):
        p = torch.from_numpy(psi.astype(dtype)).to(cuda_device)
        got = ham.apply_within(dev, p, dev).cpu().numpy()
        want = oracle.apply_within(site, kind, coef, rows, psi.astype(dtype).astype(np.complex128), rows)
        assert np.all(np.abs(got - want) <= tol * total * np.abs(psi).max())
