"""Radial tables of a planned basis: the copy for the radial-index lanes only where they run."""
import ctypes

import pytest

from cusoap_b200 import _lib


@pytest.mark.parametrize("n_max", [1, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("l_max", [0, 6, 7, 9, 12])
def test_interleaved_table(n_max, l_max):
    if l_max >= 10 and n_max > 8:
        return
    b = _lib.Basis()
    b.n_max, b.l_max, b.n_species, b.crossover, b.r_cut, b.sigma = n_max, l_max, 2, 1, 5.0, 0.5
    _lib.check(_lib.load().soapb_basis_plan(ctypes.byref(b)))
    table = lambda lanes: -(-4 * b.n_seg * lanes * (l_max + 1) * 8 // 256) * 256  # noqa: E731
    lanes = 0 if n_max > 8 or l_max > 6 else 4 if n_max <= 4 else 8
    assert b.off_tab_bh - b.off_tab_b == table(n_max) + table(lanes)
    assert (b.bytes - b.off_tab_bh) % 256 == 0
