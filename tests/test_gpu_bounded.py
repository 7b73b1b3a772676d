"""find_relative's bounded passes (groups read only as far as their norms can reach) against the oracle.

Byte-exact rows for tables in |coef| order and in shuffled order (bounds that
differ from the norms), one to three key words, inputs that are sampled and
that are not, selections of one record, of some and of all, and an exclusion
set that leaves the rows' own diagonal records in.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle
from qmb_gb300 import Hamiltonian, terms

pytestmark = pytest.mark.gpu


def _spread(rows, n_qubytes, shift):
    bits = np.unpackbits(rows, axis=1, bitorder="little")
    wide = np.zeros((rows.shape[0], 8 * n_qubytes), dtype=np.uint8)
    wide[:, shift:shift + bits.shape[1]] = bits[:, :8 * n_qubytes - shift]
    return terms.sort_rows(terms.pack_sites(wide, n_qubytes))


@pytest.mark.parametrize("n_qubytes,shift", [(2, 0), (5, 20), (9, 56), (17, 100)])
@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("n_i", [1, 333, 4100])
def test_rows_match_the_oracle(n_qubytes, shift, shuffled, n_i, cuda_device):
    n = 8
    site, kind, coef = (x.numpy() for x in terms.integral_hamiltonian_tables(n, seed=21, complex_valued=True))
    if shuffled:
        order = np.random.default_rng(1).permutation(site.shape[0])
        site, kind, coef = site[order], kind[order], coef[order]
    site = np.where(kind == 2, site, site + shift).astype(np.int16)
    pool = terms.all_determinants(n, 4, 4)
    rng = np.random.default_rng(2)
    pick = rng.permutation(pool.shape[0])
    rows = _spread(pool[np.sort(pick[:min(n_i, 4100)])], n_qubytes, shift)
    other = _spread(pool[np.sort(pick[-40:])], n_qubytes, shift)
    psi = terms.random_psi(rows.shape[0], seed=3) * np.exp(rng.standard_normal(rows.shape[0]) * 2)
    psi[::7] = 0
    ham = Hamiltonian((torch.from_numpy(site), torch.from_numpy(kind), torch.from_numpy(coef)), kind="fermi")
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to(cuda_device)
    counts = (1, 97, 5000) if n_i > 1000 else (1, 97, 10**6)
    for exclude in (None, other):
        for k in counts:
            got = ham.find_relative(dev(rows), dev(psi), k, None if exclude is None else dev(exclude)).cpu().numpy()
            want, _ = oracle.find_relative(site, kind, coef, rows, psi, k, exclude, 1, rule="ranked")
            assert np.array_equal(got, want), (k, exclude is None)
