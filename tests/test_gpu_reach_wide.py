"""The bounded tiled walks on two words whose halves both tell rows apart (the sizes that take them)."""

from __future__ import annotations

import pytest

import test_gpu_reach

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_qubytes,shift", [(14, 30), (16, 40)])
@pytest.mark.parametrize("kinds", [("random", None), ("halves", None), ("chains", None), ("chains", "halves"), ("halves", "chains")])
def test_two_wide_words(n_qubytes, shift, kinds, cuda_device):
    test_gpu_reach.test_reach_matches_the_oracle(n_qubytes, shift, kinds, cuda_device)
