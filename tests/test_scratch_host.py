"""Scratch that calls ask for, on the CPU: the pair scan's only where a call may scan."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from qmb_gb300 import _native as native
from qmb_gb300 import terms
from test_abi import compile_table


@pytest.fixture(scope="module")
def blob():
    site, kind, coef = (x.numpy() for x in terms.integral_hamiltonian_tables(10, seed=111))
    return compile_table(native.library(), site, kind, coef, 3, 1)


def _asked(blob, n_i, n_j):
    lib, out = native.library(), ctypes.c_uint64()
    sizes = {}
    native.check(lib.qmbx_apply_within_workspace(blob.ctypes.data, n_i, n_j, ctypes.byref(out)))
    sizes["apply"] = out.value
    native.check(lib.qmbx_matrix_workspace(blob.ctypes.data, n_i, ctypes.byref(out)))
    sizes["matrix"] = out.value
    native.check(lib.qmbx_hitlog_bytes(blob.ctypes.data, n_i, n_j, 0, 16, ctypes.byref(out)))
    sizes["log"] = out.value
    return sizes


@pytest.mark.parametrize("n_i,n_j", [(1, 1), (3, 7), (500, 500), (4000, 200)])
def test_calls_that_walk_ask_for_no_scan(blob, n_i, n_j, monkeypatch):
    # a row's keys, hash entries and sums are below 512 bytes on either side, and a few tables of fixed size
    monkeypatch.delenv("QMBX_WALK", raising=False)
    for name, size in _asked(blob, n_i, n_j).items():
        assert size <= 512 * (n_i + n_j) + (1 << 16), name


def test_forced_scan_asks_for_its_scratch(blob, monkeypatch):
    monkeypatch.delenv("QMBX_WALK", raising=False)
    plain = _asked(blob, 500, 400)
    monkeypatch.setenv("QMBX_WALK", "scan")
    forced = _asked(blob, 500, 400)
    for name in plain:
        assert forced[name] >= plain[name] + 8 * 500 * 400 // 2, name


def test_sizes_that_may_scan_ask_for_it_whatever_is_forced(blob, monkeypatch):
    # a backward finds the scratch that its forward had, also when the environment changed meanwhile
    monkeypatch.delenv("QMBX_WALK", raising=False)
    free = _asked(blob, 60000, 60000)
    for walk in ("grouped", "scan"):
        monkeypatch.setenv("QMBX_WALK", walk)
        assert _asked(blob, 60000, 60000) == free
    assert free["apply"] >= 8 * (1 << 22)


def _lattice_bytes(sites, n_qubytes, n):
    out = {}
    for a in range(sites - 1):
        out[((a, 1), (a + 1, 0))] = out[((a + 1, 1), (a, 0))] = -1.0
    site, kind, coef = (x.numpy() for x in terms.sort_terms(*terms.prepare(out)))
    lattice = compile_table(native.library(), site, kind, coef, n_qubytes, 1)
    size = ctypes.c_uint64()
    native.check(native.library().qmbx_apply_within_workspace(lattice.ctypes.data, n, n, ctypes.byref(size)))
    return size.value


@pytest.mark.parametrize("sites,n,bounded", [(72, 1000000, False), (80, 1000000, False), (96, 100000, False), (96, 300000, True),
                                             (112, 65535, False), (112, 65536, True), (136, 65536, True)])
def test_walks_are_bounded_where_the_other_words_tell_rows_apart(sites, n, bounded, monkeypatch):
    # the bound's filters take 32 bits a row and word, twice at most for rounding; row sets and sums of two and three
    # words are compared with those of a table that is never bounded (72 sites; 136 without its rows)
    monkeypatch.delenv("QMBX_WALK", raising=False)
    if sites > 128:
        assert bounded
        assert _lattice_bytes(sites, 17, n) - _lattice_bytes(sites, 17, n - 1) > 4 * 3 * n // 2
        return
    extra = _lattice_bytes(sites, (sites + 7) // 8, n) - _lattice_bytes(66, 9, n)
    assert (extra >= 4 * 2 * n // 2) == bounded
