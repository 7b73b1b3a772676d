"""Host logic of the Lanczos recurrence on a stored matrix, on the CPU: a stand-in does the iteration's arithmetic."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from qmb_gb300 import solvers


class DenseMatrix:
    """HamiltonianMatrix.lanczos_step on a dense matrix; counts the iterations."""

    def __init__(self, h: np.ndarray):
        self.h = torch.from_numpy(h).to(torch.complex128)
        self.val, self.n, self.steps = self.h, h.shape[0], 0

    def lanczos_step(self, v_prev, beta_prev, v, v_next, alpha, beta, scratch):
        self.steps += 1
        w = self.h @ v
        alpha.copy_((w.conj() @ v).real)
        w = w - alpha * v - (beta_prev * v_prev if v_prev is not None else 0)
        beta.copy_(torch.linalg.norm(w))
        v_next.copy_(w / beta)


def _matrix(n, seed):
    rng = np.random.default_rng(seed)
    h = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    return h + h.conj().T, rng.standard_normal(n) + 1j * rng.standard_normal(n)


def _check(energy, vector, h):
    v = vector.numpy()
    assert abs(np.vdot(v, h @ v).real / np.vdot(v, v).real - energy) <= 1e-9 * np.abs(h).sum()


@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64, torch.float64])
def test_lazy_conjugates_and_other_types(dtype):
    h, start = _matrix(40, 1)
    x = torch.from_numpy(start)
    x = x.to(dtype) if dtype.is_complex else x.real.contiguous().to(dtype)
    plain, _ = solvers._lanczos_on_matrix(DenseMatrix(h), x.conj().resolve_conj().clone(), 8, 1e-12)
    energy, vector = solvers._lanczos_on_matrix(DenseMatrix(h), x.conj(), 8, 1e-12)
    assert abs(energy - plain) <= 1e-12 * abs(plain)
    _check(energy, vector, h)
    energy, _ = solvers._lanczos_on_matrix(DenseMatrix(h), torch._neg_view(x), 8, 1e-12)
    want, _ = solvers._lanczos_on_matrix(DenseMatrix(h), -x, 8, 1e-12)
    assert abs(energy - want) <= 1e-12 * abs(want)


def test_more_steps_than_memory_has_places():
    # "until the recurrence ends": nothing is reserved for steps that are never taken
    h, start = _matrix(6, 2)
    energy, vector = solvers._lanczos_on_matrix(DenseMatrix(h), torch.from_numpy(start), 10**15, 1e-9)
    assert abs(energy - np.linalg.eigvalsh(h)[0]) <= 1e-8 * np.abs(h).sum()
    _check(energy, vector, h)


@pytest.mark.parametrize("ends", [1, 2, 3, 5, 9, 14])
@pytest.mark.parametrize("step", [0, 1, 2, 7, 12, 13, 100])
def test_few_iterations_run_past_the_end(ends, step):
    # an invariant subspace of `ends` vectors; the norm that ends the recurrence is seen within eight iterations
    h = np.zeros((20, 20), dtype=np.complex128)
    h[:ends, :ends], start = _matrix(ends, 10 + ends)
    v = np.zeros(20, dtype=np.complex128)
    v[:ends] = start
    mat = DenseMatrix(h)
    energy, vector = solvers._lanczos_on_matrix(mat, torch.from_numpy(v), step, 1e-9)
    assert mat.steps <= min(step + 2, ends + min(7, ends + 1))
    basis = min(step + 2, ends)
    q, _ = np.linalg.qr(np.stack([np.linalg.matrix_power(h[:ends, :ends] / 10, k) @ start for k in range(basis)], axis=1))
    want = np.linalg.eigvalsh(q.conj().T @ h[:ends, :ends] @ q)[0]
    assert abs(energy - want) <= 1e-6 * np.abs(h).sum()
    _check(energy, vector, h)
