"""Four-phonon counts against the oracle where the counting kernel changes: every
thread with its own sums (up to 16 branches) or one copy per warp (more), windows
found through the cell table on few and many pair sums, and a cell whose pair sums all
fall into few cells (one heavy and one light mass)."""
import numpy as np
import pytest

import helpers as H
import oracle as O
from fourphonon_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cell,grid", [("diamond", (2, 3, 5)), ("zincblende", (3, 3, 3)), ("random3", (2, 3, 3)),
                                       ("random5", (2, 2, 3)), ("random6", (2, 2, 3)), ("random7", (2, 2, 3))])
def test_counts_match_the_oracle(cell, grid):
    s = H.cached_solve(cell, grid)
    n, p = O.Oracle(s).np4()
    ctx = abi.Context(0)
    try:
        gn, gp = ctx.np_driver_4ph(s)
    finally:
        ctx.close()
    for ch in range(3):
        assert np.array_equal(gn[ch], n[ch])
        # a few thousand terms of one exponential and one reciprocal each
        assert np.all(np.abs(gp[ch] - p[ch]) <= 1e-12 * np.abs(p[ch]) + 1e-15 * np.abs(p[ch]).max())
