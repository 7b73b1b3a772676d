"""The pair scan (rows compared with rows, QMBX_WALK=scan) against the oracle.

Sizes are the edges of its tiles (4,096 or 2,048 rows of planes, 128 staged
rows, 32-row words), odd and even particle numbers (the four-position steps
and their remainder), one to four key words, mixed particle numbers, repeated
rows, one-term and many-term transitions, both directions, both precisions
and the matrix build.  FP64 results agree to 1e-12 of the absolute sum of a
row's contributions (the order of summation differs), the FP32 path to 2e-7.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle
from conftest import golden
from qmb_gb300 import Hamiltonian, terms

pytestmark = pytest.mark.gpu


def _scale(site, kind, coef, ci, psi, cj):
    mag = np.zeros_like(coef)
    mag[:, 0] = np.hypot(coef[:, 0], coef[:, 1])
    return np.abs(oracle.apply_within(site, kind, mag, ci, np.abs(psi).astype(np.complex128), cj, 2))


def _psi(n, seed):
    return terms.random_psi(n, seed=seed)


def _check(site, kind, coef, ci, cj, device, dtype, particles="fermi"):
    pc = 1 if particles == "fermi" else 2
    ham = Hamiltonian((torch.from_numpy(site), torch.from_numpy(kind), torch.from_numpy(coef)), kind=particles)
    psi = _psi(ci.shape[0], 5).astype(dtype)
    gj = _psi(cj.shape[0], 6).astype(dtype)
    tol = 1e-12 if dtype == np.complex128 else 2e-7
    di = torch.from_numpy(ci).to(device)
    dj = di if cj is ci else torch.from_numpy(cj).to(device)
    p = torch.from_numpy(psi).to(device).requires_grad_(True)
    y = ham.apply_within(di, p, dj)
    (back,) = torch.autograd.grad(y, p, grad_outputs=torch.from_numpy(gj).to(device))
    walked = ham.apply_within_adjoint(di, torch.from_numpy(gj).to(device), dj)
    want = oracle.apply_within(site, kind, coef, ci, psi.astype(np.complex128), cj, pc)
    scale = _scale(site, kind, coef, ci, psi, cj)
    assert np.all(np.abs(y.detach().cpu().numpy() - want) <= tol * scale + 1e-300)
    want = oracle.apply_within_adjoint(site, kind, coef, ci, cj, gj.astype(np.complex128), pc)
    mag = np.zeros_like(coef)
    mag[:, 0] = np.hypot(coef[:, 0], coef[:, 1])
    scale = np.abs(oracle.apply_within_adjoint(site, kind, mag, ci, cj, np.abs(gj).astype(np.complex128), 2))
    for got in (back, walked):
        assert np.all(np.abs(got.cpu().numpy() - want) <= tol * scale + 1e-300)
    return ham


@pytest.fixture(autouse=True)
def scan(monkeypatch):
    monkeypatch.setenv("QMBX_WALK", "scan")


@pytest.mark.parametrize("n_i,n_j", [(1, 1), (31, 33), (127, 129), (300, 4095), (4097, 128), (257, 4096), (400, 0)])
@pytest.mark.parametrize("alpha,beta", [(1, 0), (2, 1), (3, 2), (4, 4)])
def test_tile_edges(n_i, n_j, alpha, beta, cuda_device):
    n = 10
    space = len(terms.all_determinants(n, alpha, beta))
    n_i, n_j = min(n_i, space), min(n_j, space)
    site, kind, coef = (x.numpy() for x in terms.integral_hamiltonian_tables(n, seed=7, complex_valued=True))
    ci = terms.random_determinants(n, alpha, beta, n_i, seed=1)
    cj = terms.random_determinants(n, alpha, beta, n_j, seed=2) if n_j else ci
    for dtype in (np.complex128, np.complex64):
        _check(site, kind, coef, ci, cj, cuda_device, dtype)


@pytest.mark.parametrize("n_qubytes", [3, 8, 9, 16, 17, 25, 32])
def test_key_words(n_qubytes, cuda_device):
    # the same operators on rows of more sites, moved to the upper sites of the row
    n = 8
    site, kind, coef = (x.numpy() for x in terms.integral_hamiltonian_tables(n, seed=8, complex_valued=True))
    site = np.where(kind == 2, site, site + 8 * n_qubytes - 2 * n).astype(np.int16)
    bits = np.zeros((700, 8 * n_qubytes), dtype=np.uint8)
    low = np.unpackbits(terms.random_determinants(n, 3, 4, 700, seed=3), axis=1, bitorder="little")[:, :2 * n]
    bits[:, 8 * n_qubytes - 2 * n:] = low
    rows = terms.unique_rows(terms.pack_sites(bits, n_qubytes))
    _check(site, kind, coef, rows[::2].copy(), rows[1::3].copy(), cuda_device, np.complex128)
    _check(site, kind, coef, rows, rows, cuda_device, np.complex64)


def test_mixed_particle_numbers_and_repeats(cuda_device):
    # every number from the empty row to the full one, rows repeated on both sides
    n = 6
    site, kind, coef = (x.numpy() for x in terms.integral_hamiltonian_tables(n, seed=9))
    rows = np.concatenate([terms.all_determinants(n, a, b) for a in range(n + 1) for b in range(max(0, a - 1), a + 1)])
    rng = np.random.default_rng(4)
    ci = rows[rng.integers(0, rows.shape[0], size=700)]
    cj = rows[rng.integers(0, rows.shape[0], size=900)]
    _check(site, kind, coef, ci, cj, cuda_device, np.complex128)


def test_hard_core_bosons(cuda_device):
    # hops and pair hops with occupied-site conditions, no parity signs
    rng = np.random.default_rng(12)
    out = {}
    for _ in range(400):
        a, b, c, d = rng.choice(16, size=4, replace=False)
        out[((a, 1), (b, 1), (c, 0), (d, 0))] = complex(rng.standard_normal(), rng.standard_normal())
        out[((a, 1), (b, 0), (c, 1), (c, 0))] = complex(rng.standard_normal(), rng.standard_normal())
        out[((a, 1), (b, 0))] = complex(rng.standard_normal(), rng.standard_normal())
    site, kind, coef = (x.numpy() for x in terms.sort_terms(*terms.prepare(out)))
    rows = np.unique(rng.integers(0, 256, size=(1500, 2), dtype=np.uint8), axis=0)
    _check(site, kind, coef, rows[::2].copy(), rows, cuda_device, np.complex128, "bose2")


def test_small_record_repeats_the_scan(cuda_device):
    # a record too small for the hits: the backward scans again over the rows the forward prepared
    g = golden("ab_initio_10_complex")
    ham = Hamiltonian((torch.from_numpy(g["site"]), torch.from_numpy(g["kind"]), torch.from_numpy(g["coef"])), kind="fermi")
    ham._LOG_FIRST_GUESS = 4
    ci, cj = (torch.from_numpy(g[k]).to(cuda_device) for k in ("configs_i", "configs_j"))
    p = torch.from_numpy(g["psi_i"]).to(cuda_device).requires_grad_(True)
    gj = torch.randn(cj.shape[0], dtype=torch.complex128, device=cuda_device)
    want = ham.apply_within_adjoint(ci, gj, cj)
    for _ in range(2):
        (got,) = torch.autograd.grad(ham.apply_within(ci, p, cj), p, grad_outputs=gj)
        assert (got - want).abs().max().item() <= 1e-12 * want.abs().max().item()


@pytest.mark.parametrize("n", [5, 129, 3000])
def test_matrix(n, cuda_device):
    site, kind, coef = (x.numpy() for x in terms.integral_hamiltonian_tables(9, seed=10, complex_valued=True))
    rows = terms.random_determinants(9, 3, 3, n, seed=11)
    ham = Hamiltonian((torch.from_numpy(site), torch.from_numpy(kind), torch.from_numpy(coef)), kind="fermi")
    c = torch.from_numpy(rows).to(cuda_device)
    mat = ham.matrix(c)
    x = _psi(n, 13)
    got = mat.apply(torch.from_numpy(x).to(cuda_device)).cpu().numpy()
    want = oracle.apply_within(site, kind, coef, rows, x, rows)
    assert np.all(np.abs(got - want) <= 1e-12 * _scale(site, kind, coef, rows, x, rows) + 1e-300)
    assert torch.all(mat.col[mat.row_ptr[:-1]] == torch.arange(n, device=cuda_device))  # the diagonal comes first


def test_few_particles_are_walked(cuda_device):
    # three particles a row: the device takes the walk, in the forward, its record and the matrix
    n = 9
    site, kind, coef = (x.numpy() for x in terms.integral_hamiltonian_tables(n, seed=14, complex_valued=True))
    rows = terms.all_determinants(n, 2, 1)
    for ci, cj in ((rows[::2].copy(), rows), (rows, rows)):
        ham = _check(site, kind, coef, ci, cj, cuda_device, np.complex128)
    x = _psi(rows.shape[0], 15)
    got = ham.matrix(torch.from_numpy(rows).to(cuda_device)).apply(torch.from_numpy(x).to(cuda_device)).cpu().numpy()
    want = oracle.apply_within(site, kind, coef, rows, x, rows)
    assert np.all(np.abs(got - want) <= 1e-12 * _scale(site, kind, coef, rows, x, rows) + 1e-300)
