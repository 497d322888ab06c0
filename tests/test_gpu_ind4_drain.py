"""Ind_driver_4ph where one work item holds more processes of a branch pair than its queue,
so that phase B runs in the middle of the item's lists: a broadening that lets every
process of the lowest branch pass, against RTA_driver_4ph (whose own drains are at other
places) and the sums of the per-process Gamma."""
import dataclasses

import numpy as np
import pytest

import helpers as H
from fourphonon_b200 import abi

pytestmark = pytest.mark.gpu

DRAIN = 8192 - 8 * 256  # entries of a bin at which the queues are drained


def _one_branch():
    s = H.cached_solve("diamond", (6, 6, 6))
    w = s.wedge
    ll = 4
    q = int(w.list[ll]) - 1
    low = np.sort(s.energy[q])
    assert low[0] > 1.25 and low[1] > low[0]  # (frequencies up to 1.25 carry no weight)
    one = dataclasses.replace(w, nlist=1, list=np.ascontiguousarray(w.list[ll:ll + 1]), nequi=w.nequi[ll:ll + 1])
    return dataclasses.replace(s, wedge=one, scalebroad=1000.0, omega_max=float(0.5 * (low[0] + low[1])))


@pytest.mark.parametrize("precision,rtol", [(abi.FP4_PREC_FP64, 1e-12), (abi.FP4_PREC_MIXED_SIMT, 1e-4)])
def test_more_processes_than_a_queue(precision, rtol):
    s = _one_branch()
    ctx = abi.Context(0)
    try:
        n, _ = ctx.np_driver_4ph(s)
        ref = ctx.rta_driver_4ph(s)
        ctx.set_precision(precision)
        g = ctx.ind_driver_4ph(s, *n)
    finally:
        ctx.close()
    assert np.unique(g["ind2_pp"], return_counts=True)[1].max() > DRAIN
    for x, (ch, name) in enumerate((("pp", "plusplus"), ("pm", "plusminus"), ("mm", "minusminus"))):
        for key, r in (("rate_", "rate_"), ("wp_", "wp4_")):
            a, b = g[key + ch], ref[r + name][0]
            tol = rtol if key == "rate_" else 1e-12
            assert np.all(np.abs(a - b) <= tol * np.abs(b).max()), key + ch
        total = np.array([y.sum() for y in np.split(g["gamma_" + ch], np.cumsum(n[x])[:-1])])
        assert np.all(np.abs(total - g["rate_" + ch]) <= 1e-12 * np.abs(g["rate_" + ch]).max())
