"""The real-space Verlet list: rebuilt on the device when a particle has moved
more than half the skin; a list that does not fit falls back to the direct
cell scan.  Results must equal the oracle's all-pairs evaluation either way."""
import numpy as np
import pytest

import oracle as O
from helpers import TOL_FP64, TOL_MIXED, gpu_system, oracle_system, random_system, scales

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("skin", [1e-9, 0.02, 0.3])
def test_trajectory_with_frequent_or_rare_rebuilds(prec, skin):
    """skin 1e-9: a rebuild almost every step; 0.02: none in 30 steps; 0.3:
    many extra list entries, all filtered by the exact rc test."""
    ini, g = random_system(512, seed=51, rc_frac=0.3, noise=True, B0=0.02)
    sim = gpu_system(ini, g, prec, noise=2, seed=9)
    sim.set_neighbor_skin(skin)
    orc = oracle_system(ini, g)
    for _ in range(30):
        orc.step(g["dt"], 2, None, 9)
    sim.step(30, g["dt"])
    p, m, e = sim.get_state()
    po, mo, eo, _ = orc.get_state()
    d = np.abs(p - po)
    d = np.minimum(d, g["lBox"] - d)
    assert d.max() < (1e-13 if prec == 0 else 1e-10) * g["lBox"]
    assert np.abs(m - mo).max() < (1e-11 if prec == 0 else 1e-5)
    assert np.abs(e - eo).max() < (1e-11 if prec == 0 else 1e-5)


@pytest.mark.parametrize("prec,tol", [(0, TOL_FP64), (1, TOL_MIXED)])
def test_list_overflow_falls_back_to_cell_scan(prec, tol):
    ini, g = random_system(2000, seed=52, rc_frac=0.22)
    fAl, bAl, _ = scales(ini, g)
    sim = gpu_system(ini, g, prec)
    orc = oracle_system(ini, g)
    Bo, Fo, _ = orc.compute_interactions()
    B0, F0, _ = sim.CompInteractions()
    used = sim.neighbor_capacity()
    assert used > 0
    sim.neighbor_capacity(cap=used // 10)       # the next build cannot fit
    sim.set_state(g["pos"], g["mm"], g["ea"])
    B1, F1, _ = sim.CompInteractions()            # direct scan this time
    assert O.rms_rel(B1, Bo, bAl) < tol and O.rms_rel(F1, Fo, fAl) < tol
    sim.set_state(g["pos"], g["mm"], g["ea"])
    B2, F2, _ = sim.CompInteractions()            # grown list again
    assert sim.neighbor_capacity() == used
    assert O.rms_rel(B2, Bo, bAl) < tol and O.rms_rel(F2, Fo, fAl) < tol
    assert O.rms_rel(B0, Bo, bAl) < tol


@pytest.mark.parametrize("n,rc_frac", [(2, 0.45), (3, 0.4), (33, 0.5), (64, 0.25), (257, 0.35), (1001, 0.3),
                                       (2999, 0.2), (4096, 0.12)])
def test_lists_built_for_two_particles_at_once(n, rc_frac):
    """Mixed path: one warp lists the neighbours of two consecutive sorted
    particles (odd counts, one-cell grids, boxes that do not fit the periodic
    cell and fine grids).  Every pair within rc is found, on either path, and
    the pressure, whose terms along the own moment are taken from the field's
    sums, equals the oracle's (TOL_MIXED of a contact force times rc per
    particle)."""
    ini, g = random_system(n, seed=53 + n, rc_frac=rc_frac, lognormal=n % 2 == 1)
    fAl, bAl, _ = scales(ini, g)
    x = g["pos"]
    want = 0
    for i in range(n):
        d = x[:, i + 1:] - x[:, i:i + 1]
        d -= g["lBox"] * np.rint(d / g["lBox"])
        want += int(((d ** 2).sum(0) < g["rc"] ** 2).sum())
    Bo, Fo, Po = oracle_system(ini, g).compute_interactions()
    for prec in (0, 1):
        sim = gpu_system(ini, g, prec)
        B, F, P = sim.CompInteractions()
        assert sim.pairs() == want
        tol = TOL_MIXED if prec else TOL_FP64
        assert O.rms_rel(B, Bo, bAl) < tol and O.rms_rel(F, Fo, fAl) < tol
        np.testing.assert_allclose(P, Po, rtol=0, atol=tol * fAl * g["rc"] * n)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n,rc_frac", [(65, 0.4), (1001, 0.3), (2000, 0.25)])
def test_lists_beyond_their_share(prec, n, rc_frac):
    """A capacity of exactly the entries in use: some list is longer than an equal
    share of it, and the lists are written again one after another; the entries
    and their order, strong pairs included, are the same."""
    ini, g = random_system(n, seed=n, rc_frac=rc_frac, lognormal=True)
    sim = gpu_system(ini, g, prec)
    a = sim.CompInteractions()
    used = sim.neighbor_capacity()
    sim.neighbor_capacity(cap=used)
    sim.set_state(g["pos"], g["mm"], g["ea"])
    b = sim.CompInteractions()
    assert sim.neighbor_capacity() == used
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("n,rc_frac", [(33, 0.4), (1025, 0.3), (8191, 0.2), (8192, 0.2), (8193, 0.2)])
def test_cell_order_of_small_and_large_systems(n, rc_frac):
    """Up to 8192 particles one cluster of blocks makes the whole cell order,
    beyond them a kernel per stage: a stable counting sort either way, at the first
    step and after one that moved nothing."""
    ini, g = random_system(n, seed=n, rc_frac=rc_frac)
    sim = gpu_system(ini, g, 1)
    xb = g["pos"] / g["lBox"]
    xb = xb - np.floor(xb + 0.5)
    for _ in range(2):
        sim.CompInteractions()
        ncx, cs, perm = sim.debug_cells()
        c = np.clip(((xb + 0.5) * ncx).astype(np.int64), 0, ncx - 1)
        cell = (c[2] * ncx + c[1]) * ncx + c[0]
        np.testing.assert_array_equal(perm, np.argsort(cell, kind="stable"))
        np.testing.assert_array_equal(cs, np.concatenate([[0], np.cumsum(np.bincount(cell, minlength=ncx ** 3))]))


@pytest.mark.parametrize("n,rc_frac", [(2001, 0.2), (8500, 0.15)])
def test_particles_on_the_faces_of_the_box(n, rc_frac):
    """Particles within the rounding of the fixed-point coordinates (2^-33 box
    lengths) of a face, on each axis and both sides of it: whichever side their
    coordinate is rounded to, their neighbours list them and they their neighbours
    (one more of them on each side, well inside the range)."""
    ini, g = random_system(n, seed=n, rc_frac=rc_frac, lognormal=True)
    fAl, bAl, _ = scales(ini, g)
    L, x = g["lBox"], g["pos"]
    i = iter(np.random.default_rng(3).permutation(n))
    for a in range(3):
        for f in (0.5 - 1e-11, 0.5 * (1 - 1e-15), -(0.5 - 1e-11), 0.5 - 2.0 ** -34, 0.45, -0.45):
            for _ in range(4):
                x[a, next(i)] = f * L
    ref = gpu_system(ini, g, 0)
    B0, F0, P0 = ref.CompInteractions()
    sim = gpu_system(ini, g, 1)
    B, F, P = sim.CompInteractions()
    want = 0
    for k in range(n):
        d = x[:, k + 1:] - x[:, k:k + 1]
        d -= L * np.rint(d / L)
        want += int(((d ** 2).sum(0) < g["rc"] ** 2).sum())
    assert ref.pairs() == want
    # a pair at the cut-off itself may fall on either side in FP32
    assert abs(sim.pairs() - want) <= 2
    assert O.rms_rel(B, B0, bAl) < TOL_MIXED and O.rms_rel(F, F0, fAl) < TOL_MIXED
    # each particle: a missing neighbour is ~rc^-3 of a moment, far above FP32 rounding
    assert np.abs(B - B0).max() < 1e-4 * np.abs(B0).max()
    np.testing.assert_allclose(P, P0, rtol=0, atol=TOL_MIXED * fAl * g["rc"] * n)
