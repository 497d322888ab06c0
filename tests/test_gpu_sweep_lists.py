"""The in-order three-phonon sweep on process lists that are made up, against the oracle's
sequential sweep: what Ind_driver's lists of small cells do not reach."""
import dataclasses

import numpy as np
import pytest

import helpers as H
import oracle as O
from fourphonon_b200 import abi

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _solve(grid, natoms):
    """The wedge and symmetrizers of the diamond grid with 3 natoms branches of random
    frequencies and velocities."""
    s = H.cached_solve("diamond", grid)
    rng = np.random.default_rng(natoms)
    nb = 3 * natoms
    cr = dataclasses.replace(s.crystal, positions=np.zeros((3, natoms)), types=np.ones(natoms, dtype=np.int64),
                             masses=np.ones(1))
    return dataclasses.replace(s, crystal=cr, energy=np.asfortranarray(rng.uniform(1.0, 10.0, (s.nptk, nb))),
                               velocity=np.asfortranarray(rng.normal(size=(s.nptk, nb, 3))),
                               eig=np.zeros((s.nptk, nb, 1), dtype=np.complex128), ifc3=None, ifc4=None)


def _lists(s, n_plus, n_minus, seed):
    """Random processes, n_plus and n_minus of each mode; each mode's amplitudes sum to at
    most a quarter, so that a sweep of tau = 1 halves a difference at least."""
    rng = np.random.default_rng(seed)
    d = {}
    for k, n in (("plus", n_plus), ("minus", n_minus)):
        t = int(n.sum())
        d["ind2_" + k] = rng.integers(1, s.nptk * s.nb + 1, t, dtype=np.int32)
        d["ind3_" + k] = rng.integers(1, s.nptk * s.nb + 1, t, dtype=np.int32)
        d["gamma_" + k] = rng.uniform(0.0, 0.125, t) / np.repeat(np.maximum(n, 1), n)
    return d


def _compare(s, n_plus, n_minus, seed=1):
    lists = _lists(s, n_plus, n_minus, seed)
    tau = np.random.default_rng(seed + 1).uniform(0.5, 1.0, s.nmodes)
    ctx = abi.Context(0)
    try:
        F0 = ctx.iteration0(s, tau)
        got = ctx.iteration(s, F0.copy(), tau, n_plus, n_minus, lists)
        launches = ctx.stats()[4]
    finally:
        ctx.close()
    want = O.Oracle(s).iteration(F0.copy(), tau, n_plus, n_minus, lists)
    # a sum of n terms in another order: n eps of the terms' magnitudes, whose sum is at
    # most the largest |F|; the sweep at most doubles what a step brings in
    rtol = 2.0 * EPS * 2 * int(max(n_plus.max(), n_minus.max()) + 64)
    assert np.abs(got - want).max() <= rtol * np.abs(want).max()
    return launches


@pytest.mark.parametrize("natoms", [42, 43, 86])
def test_many_branches(natoms):
    """126, 129 and 258 branches: fewer and more than the threads of the sweep's chain."""
    s = _solve((2, 2, 2), natoms)
    n = np.random.default_rng(natoms).integers(0, 40, (2, s.nmodes)).astype(np.int32)
    _compare(s, n[0], n[1])


def test_the_same_bits_every_time():
    """The terms inside a block are listed, and summed, in a fixed order."""
    s = _solve((6, 6, 6), 2)
    n = np.random.default_rng(3).integers(300, 900, (2, s.nmodes)).astype(np.int32)
    lists = _lists(s, n[0], n[1], 5)
    tau = np.random.default_rng(4).uniform(0.5, 1.0, s.nmodes)
    ctx = abi.Context(0)
    try:
        F0 = ctx.iteration0(s, tau)
        first = ctx.iteration(s, F0.copy(), tau, n[0], n[1], lists)
        for _ in range(8):
            assert np.array_equal(ctx.iteration(s, F0.copy(), tau, n[0], n[1], lists), first)
    finally:
        ctx.close()
    _compare(s, n[0], n[1])


def _one_heavy_star(count):
    """The 6^3 diamond solve, with count absorption and count emission processes in each mode of its
    largest star (24 points) and 20 elsewhere."""
    s = _solve((6, 6, 6), 2)
    n = np.full((s.nlist, s.nb), 20, dtype=np.int32)
    ll = int(np.argmax(s.wedge.nequi))
    assert s.wedge.nequi[ll] == 24
    n[ll] = count
    return s, n.ravel()


@pytest.mark.parametrize("count", [58_000, 59_000])
def test_the_limit_of_the_listed_terms(count):
    """Just below and just above 32 Mi terms of one star, from where the sequential kernel runs."""
    assert (2 * 2 * 58_000 * 6 * 24 < 32 << 20) and (2 * 2 * 59_000 * 6 * 24 > 32 << 20)
    s, n = _one_heavy_star(count)
    _compare(s, n, n.copy())


def test_no_memory_for_the_listed_terms():
    """A sweep that finds no room for its terms (276 MB here) runs on the sequential kernel."""
    import torch

    s, n = _one_heavy_star(40_000)
    _compare(s, n, n.copy())  # with room; loads the kernels
    small = _solve((2, 2, 2), 43)
    _compare(small, np.zeros(small.nmodes, np.int32), np.zeros(small.nmodes, np.int32))
    free, _ = torch.cuda.mem_get_info()
    hog = torch.empty(free - (160 << 20), dtype=torch.uint8, device="cuda")
    try:
        assert torch.cuda.mem_get_info()[0] < 200 << 20
        _compare(s, n, n.copy())
    finally:
        del hog
        torch.cuda.empty_cache()


@pytest.mark.parametrize("grid,natoms,count,launches", [
    ((2, 2, 2), 2, 10, 3),       # all points in one block: its mark, its sums, its chain
    ((4, 4, 4), 8, 2_800, 17),   # many processes per mode: each of the eight stars by itself
    ((2, 2, 2), 2, 20_000, 1)])  # half of a star's many terms lie inside it: the sequential kernel
def test_the_size_of_the_blocks(grid, natoms, count, launches):
    s = _solve(grid, natoms)
    n = np.full(s.nmodes, count, dtype=np.int32)
    assert _compare(s, n, n.copy()) == launches
