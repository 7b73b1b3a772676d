"""single_relative by the terms in key order against the oracle: the same rows as a walk over all terms.

Calls above the size rule, one and two key words, terms of zero coefficient
(never drawn while another neighbour exists), tables smaller and larger than
the sorted list, and row sets that leave some or all rows without a neighbour
among the list's terms (those rows are walked).
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle
from qmb_gb300 import Hamiltonian, terms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("orbits,alpha,beta,n,n_qubytes,shift", [
    (14, 5, 5, 400, 4, 0),      # many more terms than the list holds
    (14, 1, 0, 14, 4, 0),       # below the rule: the walk
    (16, 1, 0, 16, 4, 0),
    (8, 4, 4, 4900, 2, 0),      # every determinant: no row has a neighbour
    (8, 4, 4, 4899, 2, 0),      # one is missing: only its neighbours have one
    (9, 2, 2, 1200, 10, 50),    # two key words
])
def test_rows_match_the_oracle(orbits, alpha, beta, n, n_qubytes, shift, cuda_device):
    site, kind, coef = (x.numpy() for x in terms.integral_hamiltonian_tables(orbits, seed=31, complex_valued=True))
    coef = coef.copy()
    coef[::5] = 0.0
    site = np.where(kind == 2, site, site + shift).astype(np.int16)
    pool = terms.all_determinants(orbits, alpha, beta) if orbits < 10 else \
        terms.random_determinants(orbits, alpha, beta, n, seed=4)
    bits = np.unpackbits(pool, axis=1, bitorder="little")[:, :2 * orbits]
    wide = np.zeros((pool.shape[0], 8 * n_qubytes), dtype=np.uint8)
    wide[:, shift:shift + 2 * orbits] = bits
    rows = terms.sort_rows(terms.pack_sites(wide, n_qubytes))
    rows = rows[np.sort(np.random.default_rng(5).permutation(rows.shape[0])[:n])]
    ham = Hamiltonian((torch.from_numpy(site), torch.from_numpy(kind), torch.from_numpy(coef)), kind="fermi")
    dev = torch.from_numpy(np.ascontiguousarray(rows)).to(cuda_device)
    for seed in (1, 2**61 + 17):
        got = ham.single_relative_seeded(dev, seed).cpu().numpy()
        want, _, _ = oracle.single_relative(site, kind, coef, rows, seed, 1)
        assert np.array_equal(got, want)
