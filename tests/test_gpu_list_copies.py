"""Process lists copied by several host threads (Ind_driver's outputs, the sweeps' inputs)
on every kind of stream, against the same calls on short lists, which are copied plainly.

The 16^3 diamond lists hold 110 MB, so that each thread uses each of its pinned slots
many times over, also where the threads wait for a context to have copied 256 MB."""
import dataclasses
import os

import numpy as np
import pytest

import helpers as H
from fourphonon_b200 import abi

pytestmark = pytest.mark.gpu

LISTS = ("ind2_plus", "ind3_plus", "gamma_plus", "ind2_minus", "ind3_minus", "gamma_minus")
PARTS = 32  # lists of a few MB each
OWN, LEGACY, PER_THREAD = 0, 1, 2  # stream handles: the context's own, cudaStreamLegacy, cudaStreamPerThread


@pytest.fixture(scope="module")
def solve():
    """The solve, its counts, and its lists put together from short ones."""
    s = H.cached_solve("diamond", (16, 16, 16))
    w = s.wedge
    c = abi.Context(0)
    try:
        n_p, n_m, _, _ = c.np_driver(s)
        parts = []
        for ll in np.array_split(np.arange(w.nlist), PARTS):
            part = dataclasses.replace(s, wedge=dataclasses.replace(
                w, nlist=len(ll), list=np.ascontiguousarray(w.list[ll]), nequi=w.nequi[ll]))
            m = (ll[:, None] * s.nb + np.arange(s.nb)).ravel()
            parts.append(c.ind_driver(part, n_p[m], n_m[m]))
        assert all(sum(p[k].nbytes for k in LISTS) < 8 << 20 for p in parts)
    finally:
        c.close()
    lists = {k: np.concatenate([p[k] for p in parts]) for k in LISTS + ("rate",)}
    assert sum(lists[k].nbytes for k in LISTS) * 3 > 256 << 20
    return s, n_p, n_m, lists


def _context(handle):
    c = abi.Context(0)
    c.set_stream(handle)
    return c


@pytest.mark.parametrize("handle", [OWN, LEGACY, PER_THREAD])
def test_lists_to_the_host(solve, handle):
    s, n_p, n_m, want = solve
    c = _context(handle)
    try:
        for _ in range(4):
            got = c.ind_driver(s, n_p, n_m)
            for k in LISTS:
                assert np.array_equal(got[k], want[k]), k
    finally:
        c.close()


@pytest.mark.parametrize("handle", [OWN, LEGACY, PER_THREAD])
def test_lists_to_the_device(solve, handle):
    """A Jacobi sweep sums in a fixed order: the same lists give the same bits.  The last
    pair changes the lists between."""
    s, n_p, n_m, lists = solve
    c = _context(handle)
    try:
        tau = np.where(lists["rate"] != 0.0, 1.0 / np.where(lists["rate"] != 0.0, lists["rate"], 1.0), 0.0)
        F = c.iteration0(s, tau)
        want = c.iteration_jacobi(s, F, tau, n_p, n_m, lists)
        for _ in range(4):
            assert np.array_equal(c.iteration_jacobi(s, F, tau, n_p, n_m, lists), want)
        twice = dict(lists, gamma_plus=2.0 * lists["gamma_plus"], gamma_minus=2.0 * lists["gamma_minus"])
        half = c.iteration_jacobi(s, F, 0.5 * tau, n_p, n_m, twice)  # 0.5 tau (v w) + tau sum
        zero = c.iteration_jacobi(s, np.zeros_like(F), tau, n_p, n_m, lists)  # tau v w, symmetrised
        scale = np.abs(want).max()
        assert np.abs(half - (want - 0.5 * zero)).max() <= 1e-13 * scale
    finally:
        c.close()


def test_one_usable_processor(solve):
    """A process bound to one processor copies plainly, and to the same lists."""
    s, n_p, n_m, want = solve
    mask = os.sched_getaffinity(0)
    c = abi.Context(0)
    try:
        os.sched_setaffinity(0, {min(mask)})
        for _ in range(3):
            got = c.ind_driver(s, n_p, n_m)
        for k in LISTS:
            assert np.array_equal(got[k], want[k]), k
    finally:
        os.sched_setaffinity(0, mask)
        c.close()
