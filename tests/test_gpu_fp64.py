"""FP64 path against the FP64 oracle at the edges of its kernels: particle
counts around the blocks, k cut-offs around the tasks of four |nx|, an
alpha r beyond the tables of the pair terms, coating potentials, cores in
contact.  Both sides sum ~n terms of the same size in another order, so the
contact-normalised differences stay far below TOL_FP64 = 1e-10."""
import numpy as np
import pytest

import oracle as O
from helpers import TOL_FP64, TOL_MIXED, gpu_system, oracle_system, random_system, scales

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,kc,rc_frac,alpha_rc", [
    (2, 2, 0.45, None), (31, 3, 0.5, None), (33, 4, 0.4, None), (130, 7, 0.3, None), (257, 8, 0.35, None),
    (96, 15, 0.25, None), (40, 31, 0.2, None), (64, 96, 0.3, None), (150, 5, 0.5, 9.0)])
def test_interactions_against_oracle(n, kc, rc_frac, alpha_rc):
    ini, g = random_system(n, seed=10 * n + kc, rc_frac=rc_frac, lognormal=n % 2 == 0)
    g["kc"] = kc
    if alpha_rc:  # the cut-off reaches beyond the tables (alpha r = 6)
        g["alpha"] = alpha_rc / g["rc"]
    fAl, bAl, _ = scales(ini, g)
    sim, orc = gpu_system(ini, g, 0), oracle_system(ini, g)
    B, F, P = sim.CompInteractions()
    Bo, Fo, Po = orc.compute_interactions()
    assert O.rms_rel(B, Bo, bAl) < TOL_FP64
    assert O.rms_rel(F, Fo, fAl) < TOL_FP64
    np.testing.assert_allclose(P, Po, rtol=0, atol=1e-10 * fAl * g["rc"] * n)
    rng = np.random.default_rng(n)
    mm = rng.standard_normal((3, n))
    mm /= np.linalg.norm(mm, axis=0)
    assert O.rms_rel(sim.CompDemagField(mm), orc.compute_field(mm), bAl) < TOL_FP64


@pytest.mark.parametrize("n,kc", [(2, 2), (9, 3), (33, 4), (130, 7), (257, 8), (513, 11), (100, 24), (2500, 5)])
def test_small_mixed_systems_by_rows(n, kc):
    """The default mixed engine takes the same k rows in FP32 for systems this
    small: against the FP64 path and the tensor cores, with the tolerances the
    engines are compared by elsewhere (FP32 rounding of the k-space sums)."""
    ini, g = random_system(n, seed=7 * n + kc, rc_frac=0.4, lognormal=n % 2 == 1)
    g["kc"] = kc
    fAl, bAl, _ = scales(ini, g)
    ref, rows, tc = (gpu_system(ini, g, p) for p in (0, 1, 1))
    tc.set_kspace_engine("tc")
    out = [s.CompInteractions()[:2] for s in (ref, rows, tc)]
    for q, al in ((0, bAl), (1, fAl)):
        assert O.rms_rel(out[1][q], out[0][q], al) < TOL_MIXED
        assert O.rms_rel(out[1][q], out[2][q], al) < 5e-6
    S0, S1 = ref.debug_structure_factor()[:, 3:], rows.debug_structure_factor()[:, 3:]
    assert np.sqrt(np.mean((S1 - S0) ** 2) / np.mean(S0 ** 2)) < 1e-6
    mm = g["mm"][:, ::-1].copy()
    assert O.rms_rel(rows.CompDemagField(mm), ref.CompDemagField(mm), bAl) < TOL_MIXED


@pytest.mark.parametrize("scale", [1.0, 0.35])
def test_contact_distances(scale):
    """Positions pulled together until cores touch or overlap: the clamped
    distance and the push follow the reference."""
    n = 96
    ini, g = random_system(n, seed=3, rc_frac=0.4)
    g["pos"] = np.ascontiguousarray(g["pos"] * scale)
    fAl, bAl, _ = scales(ini, g)
    sim, orc = gpu_system(ini, g, 0), oracle_system(ini, g)
    B, F, _ = sim.CompInteractions()
    Bo, Fo, _ = orc.compute_interactions()
    assert O.rms_rel(B, Bo, bAl) < TOL_FP64
    assert O.rms_rel(F, Fo, fAl) < TOL_FP64
    np.testing.assert_allclose(sim.get_state()[0], orc.get_state()[0], rtol=0, atol=1e-12 * g["lBox"])


@pytest.mark.parametrize("n,phi,errtol", [(9, 0.2, 1e-2), (65, 0.2, 1e-3), (300, 0.25, 1e-4), (1001, 0.25, 1e-4)])
def test_coating_pairs_of_the_mixed_path(n, phi, errtol):
    """Short-range cutoffs with none to ~110 coating pairs per particle (more than a
    warp queues), particle counts beyond whole blocks, mixed against FP64: the
    coating force itself is FP64 in both, so its sums differ by FP32 rounding."""
    ini, g = random_system(n, seed=n, rc_frac=0.4, phi=phi, min_gap=5e-10)
    ini["interactions"]["ENABLE_COATING_POT"] = "true"
    ini["short_range_interactions"]["errTolSR"] = str(errtol)
    fAl, bAl, _ = scales(ini, g)
    B0, F0, P0 = gpu_system(ini, g, 0).CompInteractions()
    B, F, P = gpu_system(ini, g, 1).CompInteractions()
    al = max(fAl, np.sqrt(np.mean(F0 ** 2)))
    assert O.rms_rel(B, B0, bAl) < TOL_MIXED
    assert O.rms_rel(F, F0, al) < TOL_MIXED
    np.testing.assert_allclose(P, P0, rtol=0, atol=TOL_MIXED * al * g["rc"] * n)
