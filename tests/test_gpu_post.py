"""Device post-processing: g(r) of a frame (md_rdf) against the numpy
restatement of the reference's script (mFiles/radial_dist_fun.m) on the
same positions, with and without the script's last-particle loop bound."""
import numpy as np
import pytest

from helpers import gpu_system, random_system
from md_sim_wolfschwenger_gb300 import analysis

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("include_last", [False, True])
@pytest.mark.parametrize("n,lognormal", [(1500, False), (700, True)])
def test_rdf_matches_script(n, lognormal, include_last):
    ini, g = random_system(n, seed=n + 7, rc_frac=0.3, phi=0.1, lognormal=lognormal)
    sim = gpu_system(ini, g, 1)
    sim.CompInteractions()  # moves nothing without overlaps; positions as uploaded
    pos, _, _ = sim.get_state()
    r0 = float(g["rMag"][0])
    x, gd, cnt = sim.rdf(bins=500, range_mag=8.0, r_mag0=r0, include_last=include_last)
    xr, gr = analysis.radial_distribution(pos, g["lBox"], r0, include_last=include_last)
    np.testing.assert_allclose(x, xr, rtol=1e-14)
    # integer pair counts: identical except where a pair sits within rounding
    # of a bin edge (then it moves to the neighbouring bin)
    mismatch = np.abs(gd - gr) > 1e-12 * gr.max()
    assert mismatch.sum() <= 2
    assert cnt.sum() > 0


@pytest.mark.parametrize("n,phi,bins,range_mag,shift", [
    (33, 0.02, 1, 9.0, 0), (257, 0.02, 7, 7.0, 0), (700, 0.02, 500, 8.0, 0), (2000, 0.05, 8192, 6.0, 0),
    (2000, 0.05, 500, 8.0, 2), (600, 0.1, 64, 20.0, 0)])
def test_rdf_routes(n, phi, bins, range_mag, shift):
    """The cell route at block edges, one bin, the most bins (where many pairs
    take the FP64 expression), particles some boxes outside (one wrap per
    axis only), and a long range (all pairs): counts as the script's, up to
    the pairs within rounding of a bin edge."""
    ini, g = random_system(n, seed=n + bins, rc_frac=0.3, phi=phi)
    pos = g["pos"].copy()
    if shift:
        pos[:, ::5] += shift * g["lBox"]
        pos[0, 1::7] += 0.3 * g["lBox"]
    g["pos"] = pos
    sim = gpu_system(ini, g, 1)
    r0 = float(g["rMag"][0])
    _, gd, cnt = sim.rdf(bins=bins, range_mag=range_mag, r_mag0=r0)
    _, gr = analysis.radial_distribution(pos, g["lBox"], r0, bins=bins, range_mag=range_mag)
    bw = range_mag * r0 / bins
    ref = np.rint(gr * (np.arange(bins) + 0.5) ** 2 * (2 * np.pi * bw ** 3 * n * n) / g["lBox"] ** 3).astype(np.int64)
    assert (np.abs(cnt.astype(np.int64) - ref) > 0).sum() <= 2
    assert np.abs(cnt.astype(np.int64).sum() - ref.sum()) <= 1 and ref.sum() > 0


@pytest.mark.parametrize("n", [1499, 1500, 2049, 6000])
@pytest.mark.parametrize("include_last", [False, True])
def test_rdf_of_a_gathered_frame(n, include_last):
    """All particles in 1/125 of the box, a few hundred in each cell: the cells are
    left for the tile pairs (from 1500 particles on), with the same counts."""
    ini, g = random_system(n, seed=n, rc_frac=0.3, phi=0.05)
    sim = gpu_system(ini, g, 1)
    L = 5.0 * g["lBox"]
    sim.set_box(L)
    sim.set_ewald(0.2 * g["alpha"], 5.0 * g["rc"], g["kc"])
    r0, bins = float(g["rMag"][0]), 300
    bw = 20.0 * r0 / bins
    for pos in (g["pos"], 5.0 * g["pos"], g["pos"]):  # gathered, spread over the box, gathered
        pos = np.ascontiguousarray(pos)
        sim.set_state(pos, g["mm"], g["ea"])
        _, gr = analysis.radial_distribution(pos, L, r0, bins=bins, range_mag=20.0, include_last=include_last)
        ref = np.rint(gr * (np.arange(bins) + 0.5) ** 2 * (2 * np.pi * bw ** 3 * n * n) / L ** 3).astype(np.int64)
        _, _, cnt = sim.rdf(bins=bins, range_mag=20.0, r_mag0=r0, include_last=include_last)
        assert (np.abs(cnt.astype(np.int64) - ref) > 0).sum() <= 2
        assert np.abs(cnt.astype(np.int64).sum() - ref.sum()) <= 1
        assert ref.sum() > 0
