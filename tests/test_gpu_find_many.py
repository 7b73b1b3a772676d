"""find_relative over more than 2^31 records of one weight.

All coefficients and amplitudes are 1, so every record falls in one bucket of
the selection and is emitted: 500,000 rows of 12 particles on 24 sites have
4,356 pair moves each, 2.18e9 records (52 GB).  Among equal weights the later
in visiting order (term, then row) come first, which gives the rows directly.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from qmb_gb300 import Hamiltonian, _native, terms

pytestmark = pytest.mark.gpu


def test_more_records_than_31_bits(cuda_device):
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info(cuda_device)
    if free < 100 << 30:
        pytest.skip("needs 100 GB of free device memory")
    pairs = np.array([(p, q) for q in range(24) for p in range(q)], dtype=np.int16)
    a, b = np.meshgrid(np.arange(len(pairs)), np.arange(len(pairs)), indexing="ij")
    there, back = pairs[a.ravel()], pairs[b.ravel()]
    apart = (there[:, :, None] != back[:, None, :]).all(axis=(1, 2))
    site = np.concatenate([there[apart], back[apart]], axis=1)
    kind = np.tile(np.array([1, 1, 0, 0], dtype=np.uint8), (site.shape[0], 1))
    coef = np.tile(np.array([1.0, 0.0]), (site.shape[0], 1))
    ham = Hamiltonian(tuple(torch.from_numpy(x) for x in (site, kind, coef)), kind="fermi")
    rng = np.random.default_rng(99)
    bits = np.zeros((500000, 24), dtype=np.uint8)
    np.put_along_axis(bits, np.argsort(rng.random((500000, 24), dtype=np.float32), axis=1)[:, :12], 1, axis=1)
    psi = torch.ones(bits.shape[0], dtype=torch.complex128, device=cuda_device)
    rows = torch.from_numpy(terms.pack_sites(bits, 3)).to(cuda_device)
    outside = torch.zeros((1, 3), dtype=torch.uint8, device=cuda_device)  # nothing leads to the empty row
    for count in (1000, 300000):
        got = ham.find_relative(rows, psi, count, outside).cpu().numpy()
        stats = _native.find_relative_stats()
        assert stats["records"] > 2**31 and stats["selected"] == count
        want, left = [], count
        for t in range(site.shape[0] - 1, -1, -1):
            p, q, r, s = site[t]
            takes = np.nonzero((bits[:, r] & bits[:, s] & (1 - bits[:, p]) & (1 - bits[:, q])).astype(bool))[0][::-1][:left]
            image = bits[takes].copy()
            image[:, [r, s]] = 0
            image[:, [p, q]] = 1
            want.append(image)
            left -= len(takes)
            if left == 0:
                break
        want = terms.unique_rows(terms.sort_rows(terms.pack_sites(np.concatenate(want), 3)))
        assert np.array_equal(got, want)
    del rows, psi
    torch.cuda.empty_cache()
