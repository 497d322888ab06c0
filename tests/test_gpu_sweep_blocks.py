"""The in-order three-phonon sweep in blocks of irreducible points against the
oracle's sequential sweep: several stars in one block, one star per block, cells
without symmetry (stars of two points), grids smaller than a block, and a point that
is listed twice in its star."""
import numpy as np
import pytest

import helpers as H
import oracle as O
from fourphonon_b200 import abi

pytestmark = pytest.mark.gpu

# sums of a few thousand terms in another order: 1e-16 each
RTOL = 1e-11


def _state(cell, grid):
    s = H.cached_solve(cell, grid)
    ctx = abi.Context(0)
    n_p, n_m, _, _ = ctx.np_driver(s)
    lists = ctx.ind_driver(s, n_p, n_m)
    rate = lists["rate"]
    tau = np.where(rate != 0.0, 1.0 / np.where(rate != 0.0, rate, 1.0), 0.0)
    return s, ctx, n_p, n_m, lists, tau


@pytest.mark.parametrize("cell,grid", [("diamond", (2, 2, 2)), ("diamond", (6, 6, 6)), ("diamond", (9, 9, 9)),
                                       ("zincblende", (3, 4, 5)), ("random3", (3, 3, 5))])
def test_sweeps_match_the_oracle(cell, grid):
    s, ctx, n_p, n_m, lists, tau = _state(cell, grid)
    try:
        o = O.Oracle(s)
        F = ctx.iteration0(s, tau)
        G = F.copy()
        for _ in range(2):
            F = ctx.iteration(s, F, tau, n_p, n_m, lists)
            G = o.iteration(G, tau, n_p, n_m, lists)
            assert np.abs(F - G).max() <= RTOL * np.abs(G).max()
    finally:
        ctx.close()


def test_a_point_listed_twice():
    s, ctx, n_p, n_m, lists, tau = _state("diamond", (4, 4, 4))
    w = s.wedge
    ll = int(np.argmax(w.nequi < s.sym.nsymm_rot))
    keep = (w.nequi.copy(), w.allequi.copy(), w.typeofsym.copy())
    try:
        k = int(w.nequi[ll])
        w.allequi[ll, k], w.typeofsym[ll, k] = w.allequi[ll, 0], w.typeofsym[ll, 0]
        w.nequi[ll] = k + 1
        F0 = ctx.iteration0(s, tau)
        F = ctx.iteration(s, F0.copy(), tau, n_p, n_m, lists)
        G = O.Oracle(s).iteration(F0.copy(), tau, n_p, n_m, lists)
        assert np.abs(F - G).max() <= RTOL * np.abs(G).max()
    finally:
        w.nequi[:], w.allequi[:], w.typeofsym[:] = keep
        ctx.close()
