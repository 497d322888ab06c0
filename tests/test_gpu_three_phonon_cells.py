"""Three-phonon counts, lists, amplitudes and rates against the oracle where the
kernel's passes end: candidate totals below one row, below one pass, and not a multiple
of either; grids with fewer points than a row has steps; odd branch counts and three
different grid edges."""
import numpy as np
import pytest

import helpers as H
import oracle as O
from fourphonon_b200 import abi

pytestmark = pytest.mark.gpu

RTOL = 1e-10  # up to a hundred classes of about 20 rounded operations per process


@pytest.mark.parametrize("cell,grid", [("diamond", (1, 1, 1)), ("diamond", (2, 2, 2)), ("diamond", (5, 5, 5)),
                                       ("zincblende", (2, 3, 5)), ("random3", (3, 3, 5)), ("random5", (2, 3, 3))])
def test_three_phonon_stage_matches_the_oracle(cell, grid):
    s = H.cached_solve(cell, grid)
    o = O.Oracle(s)
    ref_n = o.np3()
    ref = o.ind3(ref_n[0], ref_n[1])
    ctx = abi.Context(0)
    try:
        n_p, n_m, p_p, p_m = ctx.np_driver(s)
        only = ctx.ind_only_driver(s, n_p, n_m)
        got = ctx.ind_driver(s, n_p, n_m)
        rta = ctx.rta_driver(s)
    finally:
        ctx.close()
    assert np.array_equal(n_p, ref_n[0]) and np.array_equal(n_m, ref_n[1])
    for x, key in enumerate(("ind2_plus", "ind3_plus", "ind2_minus", "ind3_minus")):
        assert np.array_equal(got[key], ref[key]) and np.array_equal(only[x], ref[key])

    def close(x, y):
        y = np.asarray(y)
        return x.size == 0 or np.all(np.abs(x - y) <= RTOL * np.abs(y) + 1e-3 * RTOL * np.abs(y).max())

    assert close(p_p, ref_n[2]) and close(p_m, ref_n[3])
    for key in ("gamma_plus", "gamma_minus", "rate_plus", "rate_minus", "wp3_plus", "wp3_minus"):
        assert close(got[key], ref[key]), key
        if not key.startswith("gamma"):
            assert close(rta[key], ref[key]), key
