"""The pair scan's list of close pairs: full, and with more pairs than 32 bits count.

Pairs that find no place in the list are looked up by the scan itself; both
ways are compared with the grouped walk, whose results the oracle pins
elsewhere.  A sum of m products in another order differs by at most m 2^-52 of
the sum of their magnitudes; rows here have fewer than 14,000 products.
"""

from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

from qmb_gb300 import Hamiltonian, _native, terms

pytestmark = pytest.mark.gpu

TOL = 14000 * 2.0**-52


def _table(site, kind, coef):
    return tuple(torch.from_numpy(np.ascontiguousarray(x)) for x in (site, kind, coef))


def _magnitudes(table):
    """The operator with |coef|, without signs of exchange: its sums bound a row's products."""
    site, kind, coef = table
    return Hamiltonian((site, kind, torch.stack([coef.norm(dim=1), torch.zeros(coef.shape[0], dtype=coef.dtype)], dim=1)),
                       kind="bose2")


def _scanned(table, rows, targets, psi, device):
    """Whether a logged forward call scanned pairs (the log header's last word)."""
    lib = _native.library()
    same = int(rows is targets)
    nbytes = ctypes.c_uint64(0)
    n_i, n_j = rows.shape[0], targets.shape[0]
    _native.check(lib.qmbx_hitlog_bytes(table.h, n_i, n_j, same, 16, ctypes.byref(nbytes)))
    log = torch.empty(nbytes.value, dtype=torch.uint8, device=device)
    out = torch.empty(n_j, dtype=torch.complex128, device=device)
    _native.call("qmbx_apply_within_logged", table.h, table.d, rows.data_ptr(), psi.data_ptr(), n_i, targets.data_ptr(),
                 n_j, same, out.data_ptr(), log.data_ptr(), log.numel(), 16, torch.cuda.current_stream(device).cuda_stream)
    return bool(log[:48].cpu().numpy().view(np.int32)[11])


def _psi(n, seed, device):
    return torch.from_numpy(terms.random_psi(n, seed=seed)).to(device)


def test_more_pairs_than_places(cuda_device, monkeypatch):
    # 44,100 rows that 804 others each are close to: 17.7M pairs for 7M places, within the set and between two
    table = terms.integral_hamiltonian_tables(10, seed=91, complex_valued=True)
    ham, bound = Hamiltonian(table, kind="fermi"), _magnitudes(table)
    rows = torch.from_numpy(terms.all_determinants(10, 4, 4)).to(cuda_device)
    half = rows[::2].contiguous()
    monkeypatch.setenv("QMBX_WALK", "scan")
    assert _scanned(ham._table(cuda_device, rows.shape[1]), rows, rows, _psi(rows.shape[0], 1, cuda_device), cuda_device)
    for c_i, c_j in ((rows, rows), (half, rows), (rows, half)):
        psi, g = _psi(c_i.shape[0], 2, cuda_device), _psi(c_j.shape[0], 3, cuda_device)
        got = {}
        for walk in ("scan", "grouped"):
            monkeypatch.setenv("QMBX_WALK", walk)
            for first_guess in (1 << 25, 16):  # a whole record, and one that the backward repeats the forward for
                fresh = Hamiltonian(table, kind="fermi")
                fresh._LOG_FIRST_GUESS = first_guess
                p = psi.clone().requires_grad_(True)
                y = fresh.apply_within(c_i, p, c_j)
                (back,) = torch.autograd.grad(y, p, grad_outputs=g)
                got[walk, first_guess] = (y.detach(), back)
            got[walk, "adjoint"] = ham.apply_within_adjoint(c_i, g, c_j)
        monkeypatch.setenv("QMBX_WALK", "grouped")
        size = bound.apply_within(c_i, psi.abs().to(torch.complex128), c_j).abs()
        size_back = bound.apply_within_adjoint(c_i, g.abs().to(torch.complex128), c_j).abs()
        for first_guess in (1 << 25, 16):
            y, back = got["scan", first_guess]
            assert torch.all((y - got["grouped", 16][0]).abs() <= TOL * size)
            assert torch.all((back - got["grouped", "adjoint"]).abs() <= TOL * size_back)
        assert torch.all((got["scan", "adjoint"] - got["grouped", "adjoint"]).abs() <= TOL * size_back)
    entries = {}
    x = _psi(rows.shape[0], 4, cuda_device)
    for walk in ("scan", "grouped"):
        monkeypatch.setenv("QMBX_WALK", walk)
        mat = ham.matrix(rows)
        entries[walk] = (mat.nnz, mat.row_ptr, mat.apply(x))
    size = bound.apply_within(rows, x.abs().to(torch.complex128), rows).abs()
    assert entries["scan"][0] == entries["grouped"][0] and torch.equal(entries["scan"][1], entries["grouped"][1])
    assert torch.all((entries["scan"][2] - entries["grouped"][2]).abs() <= TOL * size)


def test_more_pairs_than_32_bits(cuda_device, monkeypatch):
    # four particles on 72 sites: 13,941 of the 1,028,790 rows are within a move of two of any row, so
    # 320,000 rows have 4.46e9 close pairs (equal rows are counted), more than 2^32
    rng = np.random.default_rng(92)
    pairs = np.array([(p, q) for q in range(72) for p in range(q)], dtype=np.int16)
    pick = np.unique(rng.integers(0, len(pairs) ** 2, size=360000))
    there, back = pairs[pick % len(pairs)], pairs[pick // len(pairs)]
    apart = (there[:, :, None] != back[:, None, :]).all(axis=(1, 2))
    site = np.concatenate([there[apart], back[apart]], axis=1)
    kind = np.tile(np.array([1, 1, 0, 0], dtype=np.uint8), (site.shape[0], 1))
    coef = np.stack([rng.standard_normal(site.shape[0]), np.zeros(site.shape[0])], axis=1)
    table = _table(site, kind, coef)
    ham, bound = Hamiltonian(table, kind="fermi"), _magnitudes(table)
    quads = torch.combinations(torch.arange(72, device=cuda_device), 4)
    bits = torch.zeros((quads.shape[0], 72), dtype=torch.uint8, device=cuda_device).scatter_(1, quads, 1)
    weight = (2 ** torch.arange(8, device=cuda_device)).to(torch.uint8)
    rows = (bits.view(-1, 9, 8) * weight).sum(dim=2).to(torch.uint8)
    few = rows[torch.from_numpy(rng.permutation(rows.shape[0])[:320000]).to(cuda_device)].contiguous()
    psi = _psi(few.shape[0], 5, cuda_device)
    monkeypatch.setenv("QMBX_WALK", "scan")
    assert _scanned(ham._table(cuda_device, 9), few, rows, psi, cuda_device)
    got = ham.apply_within(few, psi, rows)
    monkeypatch.setenv("QMBX_WALK", "grouped")
    want = ham.apply_within(few, psi, rows)
    size = bound.apply_within(few, psi.abs().to(torch.complex128), rows).abs()
    assert torch.all((got - want).abs() <= TOL * size)
