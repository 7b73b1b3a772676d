"""find_relative where few rows have most of the weight, against the walks (byte-exact).

The count of every group's first terms misses the records deep in such rows'
groups; the pass above its bucket counts them, so that about what is asked
for is emitted (twice the selection and the slack of two buckets, each an
eighth of a power of two, where the rows are sampled: the workspace's first
size holds it).  Groups that a row reaches far into are queued; one case has
more of them than places.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from qmb_gb300 import Hamiltonian, _native, terms

pytestmark = pytest.mark.gpu


def _weights(n, kind):
    psi = terms.random_psi(n, seed=121)
    at = np.arange(n)
    if kind == "falling":
        return psi * np.exp(-at / (n / 20))
    if kind == "power":
        return psi / (1 + at)
    if kind == "peak":
        psi = psi * 1e-4
        psi[n // 3] = 1.0
    return psi


def _both(ham, rows, psi, count, monkeypatch):
    got = ham.find_relative(rows, psi, count)
    stats = _native.find_relative_stats()
    with monkeypatch.context() as walked:
        walked.setenv("QMBX_WALK", "grouped")
        want = ham.find_relative(rows, psi, count)
    assert torch.equal(got, want)
    return stats


@pytest.mark.parametrize("kind", ["falling", "power", "peak", "even"])
@pytest.mark.parametrize("orbits,electrons,n,count", [(14, 5, 6000, 150000), (14, 5, 3000, 40000), (20, 6, 5000, 200000),
                                                      (38, 8, 4200, 100000)])
def test_records_emitted(orbits, electrons, n, count, kind, cuda_device, monkeypatch):
    monkeypatch.delenv("QMBX_WALK", raising=False)
    ham = Hamiltonian(terms.integral_hamiltonian_tables(orbits, seed=122), kind="fermi")
    rows = torch.from_numpy(terms.random_determinants(orbits, electrons, electrons, n, seed=123)).to(cuda_device)
    psi = torch.from_numpy(_weights(n, kind)).to(cuda_device)
    stats = _both(ham, rows, psi, count, monkeypatch)
    assert stats["records"] <= 4 * count + (1 << 16)


@pytest.mark.parametrize("n", [1, 40])
@pytest.mark.parametrize("count", [1, 3000, 3000000])
def test_more_rests_than_places(n, count, cuda_device, monkeypatch):
    # all of the records of 40 rows are asked for: about 4,000 groups of more than 16 terms for 2,560 places
    monkeypatch.delenv("QMBX_WALK", raising=False)
    ham = Hamiltonian(terms.integral_hamiltonian_tables(26, seed=124), kind="fermi")
    rows = torch.from_numpy(terms.random_determinants(26, 7, 7, n, seed=125)).to(cuda_device)
    psi = torch.from_numpy(_weights(n, "falling")).to(cuda_device)
    stats = _both(ham, rows, psi, count, monkeypatch)
    assert stats["selected"] <= count


def test_unsorted_tables_are_walked(cuda_device, monkeypatch):
    # norms that do not fall give no bounds: nothing more is emitted than by the walk
    monkeypatch.delenv("QMBX_WALK", raising=False)
    table = terms.integral_hamiltonian_tables(14, seed=126)
    order = torch.from_numpy(np.random.default_rng(127).permutation(table[0].shape[0]))
    ham = Hamiltonian(tuple(x[order] for x in table), kind="fermi")
    rows = torch.from_numpy(terms.random_determinants(14, 5, 5, 5000, seed=128)).to(cuda_device)
    psi = torch.from_numpy(_weights(5000, "even")).to(cuda_device)
    stats = _both(ham, rows, psi, 300000, monkeypatch)
    assert stats["records"] <= 4 * 300000 + (1 << 16)
