"""Edges of the integrator kernels and of the fixed-point coordinates."""
import numpy as np
import pytest

import oracle as O
from helpers import TOL_MIXED, gpu_system, oracle_system, random_system, scales

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("boxes", [1, 3000, 1 << 18])
def test_positions_outside_the_box(boxes):
    """Positions some boxes away are the same periodic system (the fold of the
    fixed-point coordinates, below and above its fast range).  Adding 2^18
    boxes moves a position by <= 2^18 2^-53 box lengths, ~1e-9 of a pair
    distance: far below the mixed path's budget."""
    ini, g = random_system(33, seed=8, rc_frac=0.4)
    fAl, bAl, _ = scales(ini, g)
    B0, F0, _ = gpu_system(ini, g, 1).CompInteractions()
    k = np.random.default_rng(1).choice([-boxes, 0, boxes], size=g["pos"].shape)
    g["pos"] = np.ascontiguousarray(g["pos"] + k * g["lBox"])
    B, F, _ = gpu_system(ini, g, 1).CompInteractions()
    assert O.rms_rel(B, B0, bAl) < TOL_MIXED and O.rms_rel(F, F0, fAl) < TOL_MIXED


@pytest.mark.parametrize("n", [2, 31, 128, 129, 300])
@pytest.mark.parametrize("precision", [0, 1])
def test_records_and_state_at_block_edges(n, precision):
    """State, m_z and MSD of drawn-noise steps for particle counts around the
    warps and blocks of the step kernels, against the oracle's Philox steps
    (mixed: increments of ~1e-2 in FP32, 3 steps)."""
    ini, g = random_system(n, seed=n, rc_frac=0.4, noise=True)
    sim = gpu_system(ini, g, precision, noise=2, seed=77)
    orc = oracle_system(ini, g)
    sim.step(3, g["dt"])
    for _ in range(3):
        orc.step(g["dt"], 2, seed=77)
    p, m, e = sim.get_state()
    po, mo, eo, _ = orc.get_state()
    tol = 1e-10 if precision == 0 else 2e-6
    assert np.abs(m - mo).max() < tol and np.abs(e - eo).max() < tol
    assert np.abs(p - po).max() < (1e-13 if precision == 0 else 1e-9) * g["lBox"]
    r = sim.records()
    d = po - g["pos"]
    d -= g["lBox"] * np.round(d / g["lBox"])
    np.testing.assert_allclose(r[-1, 1], mo[2].mean(), rtol=0, atol=tol)
    np.testing.assert_allclose(r[-1, 2:5], (d * d).mean(axis=1), rtol=1e-10 if precision == 0 else 1e-4)
    assert r.shape == (3, 8) and np.allclose(r[:, 0], np.arange(3) * g["dt"])


@pytest.mark.parametrize("prec", [0, 1])
def test_steps_in_one_graph_equal_single_steps(prec):
    """A long run goes on in graphs of several steps: the same bits as one call per
    step, with a change of dt and a remainder in between."""
    ini, g = random_system(150, seed=8, rc_frac=0.35, noise=True)
    a, b = (gpu_system(ini, g, prec, noise=2, seed=4) for _ in range(2))
    for k, dt in ((300, g["dt"]), (13, 0.5 * g["dt"]), (203, g["dt"])):
        a.step(k, dt)
        for _ in range(k):
            b.step(1, dt)
        for x, y in zip(a.get_state(), b.get_state()):
            np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("n", [150, 6001])
@pytest.mark.parametrize("prec", [0, 1])
def test_records_and_launches_of_steps_in_one_graph(prec, n):
    """The records of a step are taken beside the next one in a graph of eight: the
    same rows, as many as steps, and a kernel more per step but the last.  N = 6001:
    k space through the mesh (mixed)."""
    if n < 6000:
        ini, g = random_system(n, seed=8, rc_frac=0.35, noise=True)
    else:
        from test_gpu_parity import random_system_fast
        ini, g = random_system_fast(n, seed=8, phi=0.10, B0=0.02)
        g["rc"], g["kc"] = 0.2 * g["lBox"], 16 if prec else 5
        g["alpha"] = 3.5 / g["rc"]
    a, b = (gpu_system(ini, g, prec, noise=2, seed=4) for _ in range(2))
    k, dt = 150, g["dt"]
    a.step(k, dt)
    per = []
    for _ in range(k):
        b.step(1, dt)
        per.append(b.launches())
    ra, rb = a.records(), b.records()
    assert ra.shape == (k, 8)
    np.testing.assert_array_equal(ra, rb)
    for x, y in zip(a.get_state(), b.get_state()):
        np.testing.assert_array_equal(x, y)
    assert a.launches() == sum(per) + 7 * ((k - 128) // 8)
