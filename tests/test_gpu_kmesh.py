"""k space of large mixed systems through a mesh (md_kmesh.cu) against the FP64
path: the same CompDipInteractEwaldF / CompDipFieldEwaldF sums
(src/interaction.cpp:429-514, 588-672)."""
import numpy as np
import pytest

from helpers import gpu_system, random_system
from test_gpu_parity import random_system_fast

pytestmark = pytest.mark.gpu

# The window's error is 4e-9 (field) and 2.4e-7 (force) of the k-space part, the
# FP32 sums of ~100 terms add ~3e-7.
TOL = 1e-6


def k_part(sim, mm):
    B, F, _ = sim.CompInteractions()
    Br, Fr = sim.debug_real_part()
    k = sim.debug_structure_factor()
    return B - Br, F - Fr, k[:, 3] + 1j * k[:, 4], sim.CompDemagField(mm)


def rms(a, b):
    return np.sqrt(np.mean(np.abs(a - b) ** 2) / np.mean(np.abs(b) ** 2))


# sizes near the engine's bounds, with meshes of whole and partial bricks (M = 104, 88,
# 80, 72, 64, 56), a one-cell grid (rc = L / 2), odd counts
@pytest.mark.parametrize("n,kc,rc_frac", [(6001, 20, 0.3), (8501, 22, 0.3), (8501, 18, 0.25), (11301, 25, 0.5),
                                          (12000, 16, 0.2), (32771, 13, 0.12)])
def test_k_part_against_fp64(n, kc, rc_frac):
    ini, g = random_system_fast(n, seed=n, phi=0.10, B0=0.02)
    g["rc"], g["kc"] = rc_frac * g["lBox"], kc
    g["alpha"] = 3.5 / g["rc"]
    mm = np.roll(g["mm"], 1, axis=1)
    ref = k_part(gpu_system(ini, g, 0), mm)
    sim = gpu_system(ini, g, 1)
    sim.set_strong_pairs(0.0)  # their FP64 terms are not in the real part that is taken off
    got = k_part(sim, mm)
    assert rms(got[0], ref[0]) < TOL
    assert rms(got[1], ref[1]) < TOL
    assert rms(got[2], ref[2]) < TOL
    assert rms(got[3], ref[3]) < TOL
    again = k_part(sim, mm)
    assert all(np.array_equal(a, b) for a, b in zip(got, again))


def test_particles_far_from_their_cells():
    """A skin of rc: the bricks' particles come from all cells they may have
    drifted from; the result stays that of a fresh sort."""
    n = 20011
    ini, g = random_system_fast(n, seed=5, phi=0.10, B0=0.02)
    sim = gpu_system(ini, g, 1)
    mm = np.roll(g["mm"], 1, axis=1)
    a = k_part(sim, mm)
    sim.set_neighbor_skin(1.0)
    b = k_part(sim, mm)
    for q in (2, 3):
        assert rms(b[q], a[q]) < TOL


@pytest.mark.parametrize("n,kc", [(8501, 18), (12000, 16)])
def test_crowded_bricks(n, kc):
    """Half of the particles in 1/64 of the box: bricks with many times the
    particles that a block stages at once, and empty ones."""
    ini, g = random_system_fast(n, seed=n + 1, phi=0.02, B0=0.02)
    g["rc"], g["kc"] = 0.2 * g["lBox"], kc
    g["alpha"] = 3.5 / g["rc"]
    g["pos"][:, : n // 2] *= 0.25
    mm = np.roll(g["mm"], 1, axis=1)
    ref = k_part(gpu_system(ini, g, 0), mm)
    sim = gpu_system(ini, g, 1)
    sim.set_strong_pairs(0.0)
    got = k_part(sim, mm)
    for q in range(3):
        assert rms(got[q], ref[q]) < TOL


@pytest.mark.parametrize("prec", [0, 1])
def test_step_after_overlaps_were_pushed(prec):
    """CompInteractions moves overlapping cores apart, some of them into other cells
    and bricks; the next step takes them where they are, as a new context does."""
    n = 6001
    ini, g = random_system_fast(n, seed=31, phi=0.10, B0=0.02)
    g["rc"], g["kc"] = 0.2 * g["lBox"], 16
    g["alpha"] = 3.5 / g["rc"]
    g["pos"] = np.random.default_rng(7).uniform(-0.5, 0.5, (3, n)) * g["lBox"]
    a = gpu_system(ini, g, prec)
    a.CompInteractions()
    g["pos"] = a.get_state()[0]
    b = gpu_system(ini, g, prec)
    a.step(1, 1e-13)
    b.step(1, 1e-13)
    # the sums' order differs: FP32 rounding of a slope times dt and of the moments
    tol = 1e-11 if prec == 0 else 2e-6
    for x, y, s in zip(a.get_state(), b.get_state(), (g["lBox"], 1.0, 1.0)):
        assert np.abs(x - y).max() < tol * s


@pytest.mark.parametrize("skin", [1e-9, 0.9])
def test_field_after_the_skin_was_changed(skin):
    """A new skin holds from the next full evaluation on: a field at the last
    geometry still finds the particles that moved out of their cells within the old
    skin, and the list that was built for it."""
    n = 8501
    ini, g = random_system_fast(n, seed=17, phi=0.10, B0=0.02)
    g["rc"], g["kc"] = 0.25 * g["lBox"], 18
    g["alpha"] = 3.5 / g["rc"]
    sim = gpu_system(ini, g, 1)
    sim.set_neighbor_skin(0.3)
    sim.CompInteractions()
    perm = sim.debug_cells()[2]
    sim.set_state(g["pos"] + 0.08 * g["rc"], g["mm"], g["ea"])  # 0.14 rc, all together
    sim.step(1, 1e-14)
    np.testing.assert_array_equal(sim.debug_cells()[2], perm)  # not sorted anew
    mm = np.roll(g["mm"], 1, axis=1)
    a = sim.CompDemagField(mm)
    sim.set_neighbor_skin(skin)
    assert rms(sim.CompDemagField(mm), a) < TOL
    sim.CompInteractions()
    assert rms(sim.CompDemagField(mm), a) < TOL


def test_engine_of_the_current_parameters():
    """kspace_engine names what runs: by size, as chosen, and on the FP64 path."""
    ini, g = random_system(300, seed=1, rc_frac=0.4)
    small = gpu_system(ini, g, 1)
    assert small.kspace_engine() == "rows" and gpu_system(ini, g, 0).kspace_engine() == "rows"
    small.set_kspace_engine("simt")
    assert small.kspace_engine() == "simt"
    ini, g = random_system_fast(20011, seed=2, phi=0.10, B0=0.02)
    g["kc"] = 15
    large = gpu_system(ini, g, 1)
    assert large.kspace_engine() == "mesh" and large.kspace_tensor_cores()
    large.set_kspace_tiling(0, 1)
    assert large.kspace_engine() == "tc"
    large.set_kspace_tiling(-1, 1)
    assert large.kspace_engine() == "mesh"
    large.set_kspace_engine("tc")
    assert large.kspace_engine() == "tc"


@pytest.mark.parametrize("n,kc,grow", [(7001, 16, 6.0), (8501, 16, 3.0), (8501, 20, 8.0), (20011, 15, 30.0), (20011, 21, 5.0)])
def test_gathered_bricks_are_split(n, kc, grow):
    """All particles in the middle of the box (an edge of 1 / grow): the few bricks
    that hold them are split into parts, whose sums and particles come together
    again; spread over the box afterwards, and gathered once more."""
    ini, g = random_system_fast(n, seed=n + 5, phi=0.05, B0=0.02)
    L, rc = grow * g["lBox"], 0.12 * grow * g["lBox"]
    ref, sim = gpu_system(ini, g, 0), gpu_system(ini, g, 1)
    for s in (ref, sim):
        s.set_box(L)
        s.set_ewald(3.5 / rc, rc, kc)
    sim.set_strong_pairs(0.0)
    assert sim.kspace_engine() == "mesh"
    mm = np.roll(g["mm"], 1, axis=1)
    for pos in (g["pos"] + 0.3 * L, grow * g["pos"], g["pos"] + 0.5 * L):  # across faces at the end
        for s in (ref, sim):
            s.set_state(pos, g["mm"], g["ea"])
        got, want = k_part(sim, mm), k_part(ref, mm)
        for q in range(4):
            assert rms(got[q], want[q]) < TOL


def test_particles_out_of_their_cells_between_builds():
    """Particles that moved up to two cells since the last build, across the faces
    too, without a new one: spread and interpolation find them where they are."""
    n = 20011
    ini, g = random_system_fast(n, seed=6, phi=0.10, B0=0.02)
    g["rc"], g["kc"] = 0.2 * g["lBox"], 15
    g["alpha"] = 3.5 / g["rc"]
    sim = gpu_system(ini, g, 1)
    sim.set_neighbor_skin(1.0)
    sim.CompInteractions()
    ncx, _, perm = sim.debug_cells()
    shift = 0.055 * g["lBox"]  # along each axis: 0.095 L of the 0.1 L before a build
    assert sim.kspace_engine() == "mesh" and shift * ncx > 0.7 * g["lBox"]
    g["pos"], g["mm"] = g["pos"] + shift, np.roll(g["mm"], 1, axis=1)
    sim.set_state(g["pos"], g["mm"], g["ea"])
    fresh = gpu_system(ini, g, 1)
    sim.step(1, 1e-13)
    fresh.step(1, 1e-13)
    np.testing.assert_array_equal(sim.debug_cells()[2], perm)  # not sorted anew
    for x, y, s in zip(sim.get_state(), fresh.get_state(), (g["lBox"], 1.0, 1.0)):
        assert np.abs(x - y).max() < 2e-6 * s
    mm = np.roll(g["mm"], 1, axis=1)
    assert rms(sim.CompDemagField(mm), fresh.CompDemagField(mm)) < TOL


def test_mesh_beside_an_overflowed_list():
    """The pairs scan the cells directly while the list grows; k space is the mesh's."""
    ini, g = random_system_fast(8501, seed=9, phi=0.10, B0=0.02)
    g["rc"], g["kc"] = 0.25 * g["lBox"], 18
    g["alpha"] = 3.5 / g["rc"]
    mm = np.roll(g["mm"], 1, axis=1)
    ref = k_part(gpu_system(ini, g, 0), mm)
    sim = gpu_system(ini, g, 1)
    sim.set_strong_pairs(0.0)
    sim.CompInteractions()
    used = sim.neighbor_capacity()
    sim.neighbor_capacity(cap=used // 10)
    sim.set_state(g["pos"], g["mm"], g["ea"])
    for _ in range(2):  # with the list too short, and grown
        got = k_part(sim, mm)
        for q in range(4):
            assert rms(got[q], ref[q]) < TOL
    assert sim.neighbor_capacity() == used


def test_engines_changed_on_a_live_context():
    """Every engine after every other, with steps in between and after the context
    was in a batch: each evaluation is that of its own engine."""
    from md_sim_wolfschwenger_gb300 import Batch
    n, dt = 8501, 1e-16
    ini, g = random_system_fast(n, seed=10, phi=0.10, B0=0.02)
    g["rc"], g["kc"] = 0.25 * g["lBox"], 18
    g["alpha"] = 3.5 / g["rc"]
    mm = np.roll(g["mm"], 1, axis=1)
    ref = k_part(gpu_system(ini, g, 0), mm)
    sim = gpu_system(ini, g, 1)
    sim.set_strong_pairs(0.0)

    def check(tol):
        sim.set_state(g["pos"], g["mm"], g["ea"])  # the steps moved it
        got = k_part(sim, mm)
        for q in range(4):
            assert rms(got[q], ref[q]) < tol

    for engine in ("auto", "tc", "auto", "simt", "tc", "simt", "auto"):
        sim.set_kspace_engine(engine)
        assert sim.kspace_engine() == ("mesh" if engine == "auto" else engine)
        sim.step(2, dt)
        # tensor cores and row segments: ~1.3e-6
        check(TOL if engine == "auto" else 5e-6)
    for ring in (0, -1):
        sim.set_kspace_tiling(ring, 1)
        sim.step(2, dt)
        check(5e-6 if ring == 0 else TOL)
    a = sim.CompDemagField(mm)  # of other moments: the positions move by 1e-12 of a box
    b = Batch(1)
    b.add(sim, 3, dt)
    assert b.run(3) == 3
    # the batch's geometry, on the mesh
    assert rms(sim.CompDemagField(mm), a) < TOL
    sim.step(2, dt)
    check(TOL)
