"""Phase B of the four-phonon kernel against the oracle where its shapes change:
odd and even branch counts (the paired eigenvector loads), more cluster groups than
the staging area holds (tables built in several class ranges), tables of all branches
or of one branch at a time, and grids of few points (bins of a few processes)."""
import functools

import numpy as np
import pytest

import helpers as H
import oracle as O
from fourphonon_b200 import abi

pytestmark = pytest.mark.gpu

# relative errors of the FP64 sums (a few thousand terms of 1e-16) and of the FP32
# contraction (about 100 multiply-adds of 6e-8 per process)
CASES = [("diamond", (2, 2, 2)), ("diamond", (2, 3, 5)), ("zincblende", (2, 3, 4)), ("random3", (2, 2, 3)),
         ("random5", (2, 2, 3)), ("layered", (2, 2, 3)), ("random7", (2, 2, 3))]


@functools.lru_cache(maxsize=None)
def _oracle(cell, grid):
    return O.Oracle(H.cached_solve(cell, grid)).rta4()


@pytest.mark.parametrize("precision,rtol", [(abi.FP4_PREC_FP64, 1e-10), (abi.FP4_PREC_MIXED_SIMT, 1e-4)])
@pytest.mark.parametrize("cell,grid", CASES)
def test_rates_match_the_oracle(cell, grid, precision, rtol):
    s = H.cached_solve(cell, grid)
    ref = _oracle(cell, grid)
    ctx = abi.Context(0, precision)
    try:
        got = ctx.rta_driver_4ph(s)
    finally:
        ctx.close()
    for x, name in enumerate(("plusplus", "plusminus", "minusminus")):
        for key, r, tol in (("rate_", ref[x], rtol), ("wp4_", ref[3 + x], 1e-10)):
            a, b = got[key + name][0], np.asarray(r)
            assert np.all(np.abs(a - b) <= tol * np.abs(b) + 1e-3 * tol * np.abs(b).max()), (key + name)
