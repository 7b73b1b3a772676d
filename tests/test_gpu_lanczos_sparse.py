"""One Lanczos iteration on matrices of few entries a row (a thread a row), and right at the line.

Diagonal matrices, with hops between neighbours added up to and past a mean of
four entries a row; row counts around a warp's and a block's.  FP64 sums of at
most n values: n 2^-52 of the sums of magnitudes, and a few roundings each.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from qmb_gb300 import Hamiltonian, _native, lanczos_energy, terms
from qmb_gb300.hamiltonian import HamiltonianMatrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 257, 5000, 300001])
@pytest.mark.parametrize("entries", [1, 2, 3, 4, 5])
def test_step(n, entries, cuda_device):
    rng = np.random.default_rng(n + entries)
    cols = (np.arange(n)[:, None] + np.arange(entries)[None, :] * 7) % n
    val = rng.standard_normal((n, entries)) + 1j * rng.standard_normal((n, entries))
    val[::3] = val[::3].real
    v, prev = (rng.standard_normal(n) + 1j * rng.standard_normal(n) for _ in range(2))
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to(cuda_device)
    mat = HamiltonianMatrix(dev(np.arange(n + 1, dtype=np.int64) * entries), dev(cols.astype(np.int32).ravel()), dev(val.ravel()))
    hv = (val * v[cols]).sum(axis=1)
    size = (np.abs(val) * np.abs(v[cols])).sum(axis=1)
    scratch = torch.empty(16 * n + 40960, dtype=torch.uint8, device=cuda_device)
    eps = 2.0**-52
    for previous in (False, True):
        out = torch.empty(n, dtype=torch.complex128, device=cuda_device)
        scalars = torch.tensor([0.0, 0.0, 0.25], device=cuda_device, dtype=torch.float64)
        mat.lanczos_step(dev(prev) if previous else None, scalars[2] if previous else None, dev(v), out, scalars[0], scalars[1], scratch)
        a, b = scalars[:2].cpu().numpy()
        assert abs(a - np.vdot(hv, v).real) <= (n + 16) * eps * (size * np.abs(v)).sum()
        w = hv - a * v - (0.25 * prev if previous else 0)
        whole = size + abs(a) * np.abs(v) + np.abs(prev)
        assert abs(b - np.linalg.norm(w)) <= (n + 16) * eps * np.linalg.norm(whole)
        assert np.all(np.abs(out.cpu().numpy() * b - w) <= 64 * eps * whole)


def test_repeated_rows_whatever_the_message(cuda_device, monkeypatch):
    table = terms.integral_hamiltonian_tables(5, seed=71)
    rows = torch.from_numpy(terms.all_determinants(5, 2, 2)).to(cuda_device)
    start = torch.from_numpy(terms.random_psi(2 * rows.shape[0], seed=72)).to(cuda_device)

    class Reworded(Hamiltonian):
        def matrix(self, configs, **options):
            try:
                return super().matrix(configs, **options)
            except _native.QmbxError as error:
                raise _native.QmbxError(error.status, "some other words") from error

    twice = torch.cat([rows, rows])
    want, _ = lanczos_energy(Hamiltonian(table, kind="fermi"), twice, 6, start=start, materialize=False)
    got, _ = lanczos_energy(Reworded(table, kind="fermi"), twice, 6, start=start)
    assert abs(got - want) <= 1e-10 * abs(want)

    class Failing(Hamiltonian):
        def matrix(self, configs, **options):
            raise _native.QmbxError(_native.QMBX_ERR_ARGUMENT, "some other fault")

    with pytest.raises(_native.QmbxError, match="other fault"):
        lanczos_energy(Failing(table, kind="fermi"), rows, 6, start=start[:rows.shape[0]].contiguous())
