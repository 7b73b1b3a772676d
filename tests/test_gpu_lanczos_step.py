"""One Lanczos iteration on a stored matrix against the same arithmetic in numpy.

Row counts around a warp's, a block's and the vector passes' sizes, rows of
few and of many entries, with and without a previous vector.  Every sum runs
over at most n terms: 1e-13 times the sums of magnitudes bounds the order's
effect with room to spare.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle
from qmb_gb300 import Hamiltonian, lanczos_energy, terms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("orbits,alpha,beta,n", [(6, 1, 0, 1), (6, 2, 1, 33), (8, 3, 3, 257), (9, 4, 4, 5000)])
def test_step(orbits, alpha, beta, n, cuda_device):
    site, kind, coef = (x.numpy() for x in terms.integral_hamiltonian_tables(orbits, seed=61, complex_valued=True))
    rows = terms.random_determinants(orbits, alpha, beta, n, seed=62)
    ham = Hamiltonian((torch.from_numpy(site), torch.from_numpy(kind), torch.from_numpy(coef)), kind="fermi")
    mat = ham.matrix(torch.from_numpy(rows).to(cuda_device))
    v, prev = terms.random_psi(n, seed=63), terms.random_psi(n, seed=64)
    dev = lambda x: torch.from_numpy(x).to(cuda_device)
    scratch = torch.empty(16 * n + 40960, dtype=torch.uint8, device=cuda_device)
    hv = oracle.apply_within(site, kind, coef, rows, v, rows)
    size = np.abs(coef).sum() * np.abs(v).max()
    for previous in (False, True):
        out, scalars = torch.empty(n, dtype=torch.complex128, device=cuda_device), torch.tensor([0.0, 0.0, 0.25], device=cuda_device, dtype=torch.float64)
        mat.lanczos_step(dev(prev) if previous else None, scalars[2] if previous else None, dev(v), out, scalars[0], scalars[1], scratch)
        a, b = scalars[:2].cpu().numpy()
        want_a = np.vdot(hv, v).real
        assert abs(a - want_a) <= 1e-13 * n * size * np.abs(v).max()
        w = hv - a * v - (0.25 * prev if previous else 0)
        want_b = np.linalg.norm(w)
        assert abs(b - want_b) <= 1e-13 * (size + abs(a)) * n
        assert np.all(np.abs(out.cpu().numpy() * b - w) <= 1e-12 * (size + abs(a) * np.abs(v).max() + 1))


def test_breakdown_and_repeated_rows(cuda_device):
    # a start in an invariant subspace of two rows ends the recurrence; repeated rows fall back to walks
    out = {((0, 1), (1, 0)): 1.0, ((1, 1), (0, 0)): 1.0, ((2, 1), (2, 0)): 3.0}
    site, kind, coef = terms.sort_terms(*terms.prepare(out))
    ham = Hamiltonian((site, kind, coef), kind="fermi")
    rows = torch.tensor([[1], [2], [4]], dtype=torch.uint8, device=cuda_device)
    start = torch.tensor([1.0, 0.0, 0.0], dtype=torch.complex128, device=cuda_device)
    for step in (0, 1, 5, 40):
        energy, vector = lanczos_energy(ham, rows, step, start=start)
        assert abs(energy + 1.0) <= 1e-12
        assert abs(vector[2]) <= 1e-12 and abs(abs(vector[0]) - 0.5 ** 0.5) <= 1e-12
    twice = torch.cat([rows, rows])
    energy, _ = lanczos_energy(ham, twice, 3, start=torch.ones(6, dtype=torch.complex128, device=cuda_device))
    assert np.isfinite(energy)
