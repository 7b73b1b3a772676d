"""Callers of the engine that run on the device: Lanczos and the PT2 step.

``lanczos_energy`` restates the Lanczos iteration of qmb/rldiag.py:19-52 (and
the loop of qmb/haar.py:107-183): repeated square applications of H on a
fixed basis, the three-term recurrence on device in complex128, and the
lowest Ritz pair from SciPy's ``eigh_tridiagonal`` ('stebz').  Unlike the
reference, H is materialised once on the basis as a sparse matrix
(``Hamiltonian.matrix``) and every iteration is a sparse matrix-vector
product and two vector passes, whose scalars stay on the device
(``HamiltonianMatrix.lanczos_step``), unless the matrix would not fit the memory budget, in
which case every iteration walks the terms (``apply_within``) as the
reference does; the Krylov vectors stay in device memory (a GB300 holds
~280 GB), so no vector is copied to the host inside the loop.

``pt2_energy`` restates the Epstein-Nesbet second-order step of
qmb/pert.py:37-61: E0 = <psi|H|psi>/<psi|psi>, the connected space from
``find_relative``, H psi on it from ``apply_within`` and the denominators
from ``diagonal_term``; by default as one engine call (``Hamiltonian.pt2``)
that takes E0 from find_relative's own walk.
"""

from __future__ import annotations

import functools

import numpy as np
import scipy.linalg
import torch

from . import _native
from .hamiltonian import Hamiltonian

__all__ = ["lanczos_energy", "pt2_energy"]


def _matrix_budget(device: torch.device) -> int:
    """Entries of a materialised matrix allowed on `device`: a quarter of its free memory at 20 bytes each."""
    free, _total = torch.cuda.mem_get_info(device)
    return free // 4 // 20


def lanczos_energy(ham: Hamiltonian, configs: torch.Tensor, step: int, threshold: float = 1e-12, *,
                   start: torch.Tensor | None = None, generator: torch.Generator | None = None,
                   materialize: bool = True):
    """Lowest eigenvalue (float) and eigenvector (complex128) of H restricted to ``configs``.

    With ``materialize`` (the default) H is stored once as a sparse matrix on
    the distinct rows of ``configs`` when it fits a quarter of the free
    device memory; otherwise every iteration calls ``apply_within``.
    """
    if start is None:
        start = torch.randn([configs.size(0)], dtype=torch.complex128, device=configs.device, generator=generator)
    apply = functools.partial(ham.apply_within, configs, configs_j=configs)
    if materialize and configs.is_cuda and configs.size(0) > 0:
        try:
            mat = ham.matrix(configs, max_entries=_matrix_budget(configs.device))
        except _native.QmbxError as error:
            if error.status != _native.QMBX_ERR_ARGUMENT or torch.unique(configs, dim=0).shape[0] == configs.shape[0]:
                raise
            mat = None  # repeated rows: every iteration walks the terms
        if mat is not None and step >= 0:
            return _lanczos_on_matrix(mat, start, step, threshold)
        if mat is not None:
            apply = mat.apply
    v = [start.to(torch.complex128) / torch.linalg.norm(start)]
    alpha: list[torch.Tensor] = []
    beta: list[torch.Tensor] = []
    w = apply(v[-1])
    alpha.append((w.conj() @ v[-1]).real)
    w = w - alpha[-1] * v[-1]
    i = 0
    while True:
        norm_w = torch.linalg.norm(w)
        if norm_w < threshold:
            break
        beta.append(norm_w)
        v.append(w / beta[-1])
        w = apply(v[-1])
        alpha.append((w.conj() @ v[-1]).real)
        if i == step:
            break
        w = w - alpha[-1] * v[-1] - beta[-1] * v[-2]
        i += 1
    if len(beta) == 0:
        return alpha[0].item(), v[0]
    value, weights = _lowest(torch.stack(alpha).cpu().numpy(), torch.stack(beta).cpu().numpy())
    return value, functools.reduce(torch.add, (float(weight) * vector for weight, vector in zip(weights, v)))


def _lowest(alpha, beta):
    """Lowest eigenvalue and eigenvector of the tridiagonal matrix."""
    vals, vecs = scipy.linalg.eigh_tridiagonal(alpha, beta, lapack_driver="stebz", select="i", select_range=(0, 0))
    return float(vals[0]), vecs[:, 0]


# Iterations between two looks at most; the first looks come after 2, 6 and 14 iterations, so that seven at most run
# past the end of the recurrence.  A look is a wait of 30 us; without the early ones, a start that ends after two
# iterations cost 16 (1,000,000 rows of an entry each: 1.2 ms of products became 25).
_LOOK_EVERY = 8
# rows up to which vectors are allocated 16 at a time (64 MB at most); more rows take as many as there are so far
_SMALL_ROWS = 1 << 18


def _lanczos_on_matrix(mat, start: torch.Tensor, step: int, threshold: float):
    """The recurrence on a stored matrix: its scalars stay on the device, and the host looks for a norm
    below the threshold every few iterations (what ran past it is dropped)."""
    n, device = mat.n, start.device
    if start.shape != (n,) or device != mat.val.device:
        raise RuntimeError(f"start must have shape [{n}] and be on the matrix's device.")
    scratch = torch.empty(16 * n + 40960, dtype=torch.uint8, device=device)
    start = start.to(torch.complex128).resolve_conj().resolve_neg()
    first = start / torch.linalg.norm(torch.view_as_real(start))
    blocks = [first.reshape(1, n).contiguous()]
    seen = []
    v, v_prev, beta_prev, done, stop = blocks[0][0], None, None, 0, None
    room = 0  # vectors that the last of `blocks` still has room for
    # iteration k forms alpha[k], beta[k] and vector k + 1; the last one's beta and vector are not used
    while done < step + 2 and stop is None:
        count = min(done + 2, _LOOK_EVERY, step + 2 - done)
        scalars = torch.empty((2, count), dtype=torch.float64, device=device)  # alpha and beta of the iterations
        for k in range(count):
            if room == 0:
                room = 16 if n <= _SMALL_ROWS else min(16, max(1, done + k))
                blocks.append(torch.empty((room, n), dtype=torch.complex128, device=device))
            v_next = blocks[-1][-room]
            mat.lanczos_step(v_prev, beta_prev, v, v_next, scalars[0, k], scalars[1, k], scratch)
            v_prev, v, beta_prev, room = v, v_next, scalars[1, k], room - 1
        seen.append(scalars.cpu().numpy())
        small = np.nonzero(seen[-1][1] < threshold)[0]
        if len(small) and done + small[0] < step + 1:
            stop = int(done + small[0])
        done += count
    used = (step + 1 if stop is None else stop) + 1  # vectors 0 .. used - 1
    host = np.concatenate(seen, axis=1)[:, :used]
    if used == 1:
        return float(host[0, 0]), blocks[0][0]
    value, weights = _lowest(host[0], host[1, :used - 1])
    weights = torch.from_numpy(weights.astype(np.complex128)).to(device)
    result, at = torch.zeros(n, dtype=torch.complex128, device=device), 0
    for block in blocks:
        part = block[:max(0, used - at)]
        if part.shape[0]:
            result += weights[at:at + part.shape[0]] @ part
        at += block.shape[0]
    return value, result


def pt2_energy(ham: Hamiltonian, configs: torch.Tensor, psi: torch.Tensor, count_selected: int, *,
               fused: bool = True):
    """(E0, E2): the variational energy of psi and its second-order correction over the connected space.

    ``fused`` (the default) runs the step as one engine call (``Hamiltonian.pt2``:
    E0 summed by find_relative's emission pass, everything on the device);
    ``fused=False`` composes the four operators as qmb/pert.py:37-61 does.
    """
    if fused and count_selected > 0 and configs.is_cuda:
        e0, e2, _ = ham.pt2(configs, psi, count_selected)
        return e0, e2
    psi = psi.to(torch.complex128)
    energy0 = ((psi.conj() @ ham.apply_within(configs, psi, configs)) / (psi.conj() @ psi)).real.item()
    other = ham.find_relative(configs, psi, count_selected, configs)
    hpsi = ham.apply_within(configs, psi, other)
    numerator = (hpsi.conj() * hpsi).real / (psi.conj() @ psi).real
    denominator = energy0 - ham.diagonal_term(other).real
    return energy0, (numerator / denominator).sum().item()
