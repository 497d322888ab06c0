"""The sampled four-phonon estimator in FP64 where its kernel branches, against the oracle
drawing the same samples: lanes that weigh three to eight temperatures, items that keep
more processes than their list holds, and cells with more clusters than the table of the
item's mode has room for."""
import dataclasses

import numpy as np
import pytest

import helpers as H
import oracle as O
from fourphonon_b200 import abi
from fourphonon_b200 import crystal as C
from fourphonon_b200 import system as S

pytestmark = pytest.mark.gpu

CHANNELS = ("plusplus", "plusminus", "minusminus")
# the FP64 bar of the rates: sums of a few hundred V(4) terms and a few thousand processes
RTOL = 1e-10


def _compare(s, nsamples, seed, temperatures):
    ctx = abi.Context(0)
    try:
        g = ctx.rta_driver_4ph_sample(s, nsamples, seed, temperatures=temperatures)
        kept = ctx.stats()[0]
        ctx.np_driver_4ph_sample(s, nsamples, seed)
        assert ctx.stats()[0] == kept  # the counting call draws the same
    finally:
        ctx.close()
    for t, T in enumerate(temperatures):
        o = O.Oracle(s, T=T).sample4(nsamples, seed, mode=2)
        for ch, name in enumerate(CHANNELS):
            for key, ref in (("rate_", o["rate"][ch]), ("wp4_", o["wp"][ch])):
                a = g[key + name][t]
                assert np.all(np.abs(a - ref) <= RTOL * np.abs(ref) + 1e-3 * RTOL * np.abs(ref).max()), (T, key + name)
    return kept


@pytest.mark.parametrize("nT", [3, 4, 5, 8])
def test_a_lane_for_each_temperature(nT):
    s = H.cached_solve("diamond", (4, 4, 4))
    _compare(s, 5_000, 12, [100.0 * (t + 1) for t in range(nT)])


@pytest.mark.parametrize("nT", [1, 3])
def test_items_that_empty_their_list(nT):
    """Every energy passes (a broadening of 1000), so that a third of the draws survive: an item
    of 4,096 draws keeps more processes than its list's 1,024."""
    s = dataclasses.replace(H.cached_solve("diamond", (4, 4, 4)), scalebroad=1000.0)
    ns = 40_000
    kept = _compare(s, ns, 3, [300.0 + 200.0 * t for t in range(nT)])
    assert kept > 3 * s.nmodes * ns / 4  # more than 1,024 of an item's 4,096


@pytest.mark.parametrize("shell,nT", [(3, 1), (3, 3), (4, 1)])
def test_more_clusters_than_the_table_holds(shell, nT):
    """430 and 2,422 quartic clusters; the table holds 398."""
    s = S.build_solve(C.layered_rhombohedral(), (2, 2, 2), (300.0,), 20240602, fc3_shell=2, fc4_shell=shell)
    assert s.ifc4.ntri > 398
    _compare(s, 20_000, 5, [300.0 + 200.0 * t for t in range(nT)])


@pytest.mark.parametrize("cell,nsamples", [("random7", 100), ("random7", 5_000), ("diamond", 100)])
def test_items_with_few_or_no_survivors(cell, nsamples):
    """The table of the item's mode is built for an item's first survivor."""
    s = H.cached_solve(cell, (2, 2, 2))
    kept = _compare(s, nsamples, 9, [300.0])
    assert kept < 3 * s.nmodes * nsamples
