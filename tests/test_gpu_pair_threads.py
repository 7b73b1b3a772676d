"""Pair scans of rows of different widths from two host threads at once.

Both widths are one key word, so both run the same kernel, whose limit of
shared memory belongs to the kernel: neither thread's calls may change what
the other's launches may take.
"""

from __future__ import annotations

import threading

import numpy as np
import pytest
import torch

from qmb_gb300 import Hamiltonian, terms

pytestmark = pytest.mark.gpu


def test_two_widths_at_once(cuda_device, monkeypatch):
    monkeypatch.setenv("QMBX_WALK", "scan")
    table = terms.integral_hamiltonian_tables(8, seed=95)
    low = terms.random_determinants(8, 4, 4, 600, seed=96)
    work, errors = [], []
    for n_qubytes in (2, 8):
        rows = np.zeros((low.shape[0], n_qubytes), dtype=np.uint8)
        rows[:, :low.shape[1]] = low
        ham = Hamiltonian(table, kind="fermi")
        c = torch.from_numpy(rows).to(cuda_device)
        psi = torch.from_numpy(terms.random_psi(low.shape[0], seed=97)).to(cuda_device)
        work.append((ham, c, psi, ham.apply_within(c, psi, c)))
    start = threading.Barrier(2)

    def call(ham, c, psi, want):
        try:
            with torch.cuda.stream(torch.cuda.Stream(cuda_device)):
                start.wait()
                for _ in range(3000):
                    got = ham.apply_within(c, psi, c)
                assert (got - want).abs().max().item() <= 1e-12 * want.abs().max().item()
        except BaseException as error:  # the main thread reports it
            errors.append(error)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=call, args=item) for item in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
