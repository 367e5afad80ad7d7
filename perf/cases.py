"""The calls whose speed counts: what a program built on this framework has it
do, from the smallest system to the largest.

A case is a dict of plain values with a `kind`:
  step      a run of `steps` Heun steps of one system, then its state;
  step_io   one step of a system whose state stays in the caller's pinned host
            arrays between the steps;
  fields    demagnetising field and force of positions and moments that another
            integrator hands over (CompInteractions), and the field of other
            moments at the same positions (CompDemagField);
  adaptive  a run of accepted steps with the configuration's adaptive solver;
  sweep     packed steps of several systems of uneven size;
  rdf       the radial distribution function of a frame.
Systems are magnetite suspensions of the benchmark's kind (log-normal or equal
cores of 20-25 nm, 5 nm shell), except `shipped`, the reference's own
configuration file.  States come back as the library holds them: positions in
64 bits; moments and easy axes, and the mixed path's fields and forces, in the
32 bits that the mixed path computes them in.
"""
import functools
import math

import numpy as np
import torch

import md_sim_wolfschwenger_gb300 as md

DT = 1e-12
DEV = torch.device("cuda" if torch.cuda.is_available() else "cpu")


def listed():
    return [
        # the reference's CPU-size case: latency and launches of a small system
        dict(name="step_small", kind="step", n=512, sigma=0.0, phi=0.05, b0=0.01, prec="mixed", steps=100),
        # an everyday polydisperse run of a size that fills no tile
        dict(name="step_ragged", kind="step", n=3001, sigma=0.2, phi=0.10, b0=0.02, prec="mixed", steps=20),
        # the benchmark's single large instance
        dict(name="step_large", kind="step", n=32768, sigma=0.2, phi=0.10, b0=0.02, prec="mixed", steps=5),
        # the benchmark's stress instance: dense, strongly polydisperse
        dict(name="step_stress", kind="step", n=131072, sigma=0.25, phi=0.20, b0=0.03, prec="mixed", steps=2),
        # a host program that owns the state and calls the library once a step
        dict(name="step_host_state", kind="step_io", n=32768, sigma=0.2, phi=0.10, b0=0.02, prec="mixed"),
        # an external integrator that asks for fields and forces
        dict(name="fields_mixed", kind="fields", n=20011, sigma=0.2, phi=0.10, b0=0.02, prec="mixed"),
        # the same on the plain 64-bit path, used to check the mixed one
        dict(name="fields_fp64", kind="fields", n=4099, sigma=0.2, phi=0.10, b0=0.02, prec="fp64"),
        # a 64-bit trajectory
        dict(name="step_fp64", kind="step", n=1000, sigma=0.0, phi=0.05, b0=0.01, prec="fp64", steps=10),
        # the reference's configuration file as it is shipped: 1000 particles, Dormand-Prince, in 64 bits
        # like the reference (its 1e-7 Ewald tolerance is finer than the mixed path)
        dict(name="adaptive_shipped", kind="adaptive", n=1000, solver=2, coat=0, prec="fp64", steps=5, shipped=1),
        # coated particles under Heun-Euler control
        dict(name="adaptive_coated", kind="adaptive", n=2744, solver=0, coat=1, prec="mixed", steps=5, shipped=0),
        # a magnetisation curve: independent systems advanced together
        dict(name="sweep", kind="sweep", systems=32, lo=256, hi=8192, phi=0.05, steps=5),
        # analysis of a frame of the large instance
        dict(name="rdf_large", kind="rdf", n=32768, sigma=0.2, phi=0.10, bins=500),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "step_io", "fields", "fields", "fp64", "adaptive", "sweep", "rdf"])
    sigma = round(rng.choice([0.0, rng.uniform(0.05, 0.25)]), 3)
    phi = round(rng.uniform(0.02, 0.20), 3)
    b0 = round(rng.uniform(0.0, 0.05), 4)
    if kind == "step":
        n = _log_uniform(rng, 256, 131072)
        return dict(kind="step", n=n, sigma=sigma, phi=phi, b0=b0, prec="mixed", steps=max(1, min(100, 200000 // n)))
    if kind == "step_io":
        return dict(kind="step_io", n=_log_uniform(rng, 1000, 65536), sigma=sigma, phi=phi, b0=b0, prec="mixed")
    if kind == "fields":
        return dict(kind="fields", n=_log_uniform(rng, 256, 65536), sigma=sigma, phi=phi, b0=b0, prec="mixed")
    if kind == "fp64":
        n = _log_uniform(rng, 256, 8192)
        if rng.random() < 0.5:
            return dict(kind="fields", n=n, sigma=sigma, phi=phi, b0=b0, prec="fp64")
        return dict(kind="step", n=n, sigma=sigma, phi=phi, b0=b0, prec="fp64", steps=max(1, min(10, 10000 // n)))
    if kind == "adaptive":
        coat, solver = rng.randint(0, 1), rng.randint(0, 2)
        # the embedded errors of orders 3 and 5 are differences that want 64-bit slopes
        prec, top = ("mixed", 8000) if solver == 0 else ("fp64", 2744)
        return dict(kind="adaptive", n=_log_uniform(rng, 343, top), solver=solver, coat=coat, prec=prec, steps=rng.randint(2, 6),
                    shipped=0)
    if kind == "sweep":
        return dict(kind="sweep", systems=rng.randint(4, 40), lo=256, hi=8192, phi=round(rng.uniform(0.02, 0.10), 3),
                    steps=rng.randint(2, 6))
    return dict(kind="rdf", n=_log_uniform(rng, 1000, 65536), sigma=sigma, phi=phi, bins=rng.randint(100, 1000))


# ------------------------------------------------------------------ inputs


def _config(case, n, seed, b0):
    cfg = md.Configuration.default()
    if case.get("shipped"):
        cfg.set(numbPartOverride=n, seed=seed)
        return cfg
    coat = case.get("coat", 0)
    sigma = case.get("sigma", 0.0)
    cfg.set(SIZE_DIST=1 if sigma > 0 else 0, rMagMean=1e-8 if sigma < 0.25 else 1.25e-8, sigmaLog=sigma, dShell=5e-9,
            volFrac=case.get("phi", 0.05), magFluxDens=b0, tMag=1.0, satMag=4.8e5, anisEn=1.1e4, magDamp=0.1, visOverride=1e-3,
            numbPartOverride=n, errTolEwald=1e-5, seed=seed, SOLVER=case.get("solver", 0), ENABLE_COATING_POT=coat,
            INIT_CONFIG_ROT=4, noise=md.MD_NOISE_PHILOX)
    return cfg


def _precision(case):
    return md.MD_PREC_FP64 if case.get("prec") == "fp64" else md.MD_PREC_MIXED


def _system(case, n, seed, b0):
    """A new system as a program sets it up: particles, state, Ewald split."""
    cfg = _config(case, n, seed, b0)
    rMag, rHydr, pos, mm, ea, _ = md.init_system(cfg, n, seed)
    sim = md.Simulation(cfg, n, _precision(case), rMag=rMag, rHydr=rHydr)
    sim.set_ewald(*sim.ewald_params()[:3])
    sim.set_state(pos, mm, ea)
    sim.set_noise(md.MD_NOISE_PHILOX, seed)
    return dict(sim=sim, cfg=cfg, rMag=rMag, rHydr=rHydr, state=(pos, mm, ea))


def _moments(n, seed):
    """Unit moment directions, uniform on the sphere (3, n)."""
    v = np.random.default_rng(seed).standard_normal((3, n))
    return v / np.linalg.norm(v, axis=0)


def _sweep_sizes(case, seed):
    # the sizes belong to the case; the seed draws the particles
    ns = np.random.default_rng(1000 * case["systems"] + case["steps"]).integers(case["lo"], case["hi"] + 1, case["systems"])
    return [(int(n), float(b), 100 * seed + i) for i, (n, b) in enumerate(zip(ns, np.linspace(0.0, 0.05, len(ns))))]


def _pinned(n):
    return [torch.empty((3, n), dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy() for _ in range(3)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sweep":
        members = [_system(case, n, s, b) for n, b, s in _sweep_sizes(case, seed)]
        batch = md.Batch(len(members))
        for m in members:
            batch.add(m["sim"], 10 ** 5, DT)
        return dict(case=case, batch=batch, members=members)
    s = _system(case, case["n"], seed, case.get("b0", 0.0))
    s["case"] = case
    if kind == "step_io":
        s["io"] = _pinned(case["n"])
        for a, b in zip(s["io"], s["state"]):
            a[:] = b
    if kind == "fields":
        s["other"] = _moments(case["n"], seed)
    return s


# --------------------------------------------------------------------- run


def _as_held(case, state):
    """Positions in 64 bits; the mixed path's moments and axes are 32-bit values."""
    pos, mm, ea = state
    if case.get("prec") == "fp64":
        return [pos, mm, ea]
    return [pos, mm.astype(np.float32), ea.astype(np.float32)]


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "step":
        s["sim"].step(case["steps"], DT)
        return _as_held(case, s["sim"].get_state())
    if kind == "step_io":
        s["sim"].step_io(s["io"], 1, DT, out=s["io"])
        return _as_held(case, s["io"])
    if kind == "fields":
        sim = s["sim"]
        sim.set_state(*s["state"])
        B, F, _ = sim.CompInteractions()
        B2 = sim.CompDemagField(s["other"])
        out = [B, F, B2]
        return out if case["prec"] == "fp64" else [x.astype(np.float32) for x in out]
    if kind == "adaptive":
        dt, done = s["sim"].step_adaptive(case["steps"], DT)
        # the next trial step comes from a difference of slopes that all but cancel: a control value of few digits
        return _as_held(case, s["sim"].get_state()) + [np.float32(dt), done]
    if kind == "sweep":
        s["batch"].run(case["steps"])
        got = [m["sim"].get_state() for m in s["members"]]
        return _as_held(case, [np.concatenate([g[q] for g in got], axis=1) for q in range(3)])
    _, g, counts = s["sim"].rdf(case["bins"], 8.0, r_mag0=1e-8)
    return [g, counts.astype(np.int64)]


# -------------------------------------------------------------------- work


@functools.lru_cache(maxsize=64)
def _split(key, n):
    """(rc / L, kc, k vectors of the half space) of a case's system."""
    case = dict(key)
    s = _system(case, n, 1, case.get("b0", 0.0))
    _, rc, kc = s["sim"].ewald
    x = rc / s["sim"].lBox
    s["sim"].close()
    r = np.arange(-kc, kc + 1)
    inside = (r[:, None, None] ** 2 + r[None, :, None] ** 2 + r[None, None, :] ** 2 <= kc * kc).sum()
    return x, kc, (int(inside) - 1) // 2


def _evaluation(case, n):
    """Flops of one field + force and of one field evaluation of the Ewald sums:
    113 / 58 per pair within the cut-off, 32 / 23 per k vector and particle."""
    x, _, nk = _split(tuple(sorted((k, v) for k, v in case.items() if k != "name")), n)
    pairs = 0.5 * n * n * 4.0 / 3.0 * math.pi * x ** 3
    return 113.0 * pairs + 32.0 * nk * n, 58.0 * pairs + 23.0 * nk * n


def work(case):
    kind = case["kind"]
    if kind == "rdf":
        n = case["n"]
        return {"bytes": 24.0 * n + 16.0 * case["bins"], "flops": 12.0 * 0.5 * n * n * min(1.0, 4.2 * 512.0 * 1e-24 / _box(case) ** 3)}
    if kind == "sweep":
        flops = size = 0.0
        for n, _, _ in _sweep_sizes(case, 1):
            nb = 1 << (n - 1).bit_length()  # one split per power of two is near enough
            f, g = _evaluation(case, nb)
            flops += (f + g) * n / nb
            size += n
        return {"bytes": 2 * 72.0 * size, "flops": flops * case["steps"]}
    n = case["n"]
    full, field = _evaluation(case, n)
    if kind == "fields":
        return {"bytes": 168.0 * n, "flops": full + field}
    if kind == "adaptive":
        return {"bytes": 144.0 * n, "flops": case["steps"] * (full + {0: 1, 1: 3, 2: 6}[case["solver"]] * field)}
    return {"bytes": 144.0 * n, "flops": case.get("steps", 1) * (full + field)}


def _box(case):
    s = _system(case, case["n"], 1, 0.0)
    L = s["sim"].lBox
    s["sim"].close()
    return L


# ------------------------------------------------- the same in 64 bits, plain


def _fold(d, L):
    """Into the box: one wrap per axis."""
    return d - L * (d > L / 2).to(d.dtype) + L * (d < -L / 2).to(d.dtype)


class _Plain:
    """The model in torch float64: all pairs, all k vectors, arrays (3, n)."""

    def __init__(self, s, seed):
        f = lambda x: torch.as_tensor(np.ascontiguousarray(x), dtype=torch.float64, device=DEV)
        c = s["cfg"].c
        self.c, self.seed, self.t, self.stepno = c, seed, 0.0, 0
        self.pos, self.mm, self.ea = (f(x).clone() for x in s["state"])
        self.rm, rh = f(s["rMag"]), f(s["rHydr"])
        self.n, pi = len(s["rMag"]), c.my_pi
        self.L = float((4.0 / 3.0 * pi * rh ** 3).sum() / c.volFrac) ** (1.0 / 3.0)
        self.al, self.rc, self.kc = s["sim"].ewald
        vol = 4.0 / 3.0 * pi * self.rm ** 3
        vis = c.visOverride if c.visOverride > 0 else c.vis
        self.mag, self.zr, self.zt, self.vol = c.satMag * vol, 8 * pi * vis * rh ** 3, 6 * pi * vis * rh, vol
        self.v1, self.v2 = 2.0 * c.anisEn * vol / self.zr, 1.0 / self.zr
        if c.ENABLE_COATING_POT:
            self._short_range()

    def _short_range(self):
        c, r = self.c, float(self.rm.max())
        c1 = 128 * c.hamaker * r ** 6 * c.my_pi / (18 * c.mu0 * float(self.mag.max()) ** 2)
        x = 2.2 * r
        f = lambda x: c1 * x / (x * x - 4 * r * r) ** 2 - c.errTolSR
        for _ in range(1000):
            x -= f(x) / (c1 * (4 * r * r + 3 * x * x) / (4 * r * r - x * x) ** 3)
            if abs(f(x)) <= 1e-7:
                break
        self.rsr = x

    def pairs(self, mu, force):
        """Real-space sums over every ordered pair within rc."""
        c, n, al, L = self.c, self.n, self.al, self.L
        B, F = torch.zeros_like(mu), torch.zeros_like(mu)
        rows = max(1, int(2.5e7 // n))
        for a in range(0, n, rows):
            d = _fold(self.pos[:, None, :] - self.pos[:, a:a + rows, None], L)
            r2 = (d * d).sum(0)
            r2[torch.arange(r2.shape[0], device=DEV), torch.arange(a, a + r2.shape[0], device=DEV)] = 2 * L * L
            i, j = torch.nonzero(r2 < self.rc * self.rc, as_tuple=True)
            d, r2 = d[:, i, j], r2[i, j]
            i = i + a
            r = torch.sqrt(r2)
            t = 2.0 * al * torch.exp(-al * al * r2) * c.irPi / r2
            a1 = torch.erfc(al * r) / (r2 * r) + t
            a2 = 3.0 * a1 / r2 + 2.0 * al ** 2 * t
            mi, mj = mu[:, i], mu[:, j]
            d2 = (mj * d).sum(0)
            B.index_add_(1, i, c.facEwald * (a2 * d2 * d - a1 * mj))
            if not force:
                continue
            a3 = 5.0 * a2 / r2 + 4.0 * al ** 4 * t
            d1, m12 = (mi * d).sum(0), (mi * mj).sum(0)
            v = c.facEwald * ((a2 * m12 - a3 * d1 * d2) * d + a2 * (d2 * mi + d1 * mj))
            if c.ENABLE_COATING_POT:
                w = r < self.rsr
                ri, rj, rw = self.rm[i[w]], self.rm[j[w]], r[w]
                lo = i[w] < j[w]
                ra, rb = torch.where(lo, ri, rj), torch.where(lo, rj, ri)
                dd = 2 * (ra + c.effLenSurfMol)
                s = torch.where(rw <= dd, 2 * rb / (ra + rb) * c.sterRepFac * ra ** 2 * torch.log(dd / rw), 0.0)
                s = s + ri * rj / (ri + rj) * c.electrostatRepFac * torch.exp(-c.kappa * (rw - ri - rj))
                s = s - c.hamaker * rw * (4 * ri * rj) ** 3 / (
                    6 * ((rw - ri - rj) * (rw + ri + rj)) ** 2 * (rw * rw - (ri - rj) ** 2) ** 2)
                v[:, w] += s * d[:, w] / rw
            F.index_add_(1, i, -v)
        return B, F

    def waves(self, mu, force):
        """Reciprocal sums over the k vectors |n| <= kc, nz >= 0, and the self and surface terms."""
        c, L, kc, pi = self.c, self.L, self.kc, self.c.my_pi
        q = torch.arange(-kc, kc + 1, dtype=torch.float64, device=DEV)
        nx, ny, nz = torch.meshgrid(q, q, q[kc:], indexing="ij")
        n2 = nx * nx + ny * ny + nz * nz
        e = torch.where((n2 > 0) & (n2 <= kc * kc), 2.0 * torch.exp(-(pi / (self.al * L)) ** 2 * n2) / n2.clamp(min=1), 0.0)
        e = torch.where(nz == 0, 0.5 * e, e)
        k = torch.stack([nx, ny, nz]).reshape(3, 2 * kc + 1, -1).to(torch.complex128)
        e = e.reshape(2 * kc + 1, -1)
        S = torch.zeros_like(k[0])
        tables = []
        for a in range(0, self.n, 4096):
            ph = 2.0 * pi * self.pos[:, a:a + 4096] / L
            x, y, z = (torch.exp(1j * p[:, None] * (q if b < 2 else q[kc:])) for b, p in enumerate(ph))
            tables.append((x, y, z))
            yz = (y[:, :, None] * z[:, None, :]).reshape(x.shape[0], -1)
            for b in range(3):
                S += k[b] * ((x * mu[b, a:a + 4096, None]).T @ yz)
        eS = e * S
        B, F = torch.empty_like(mu), torch.zeros_like(mu)
        for t, (x, y, z) in enumerate(tables):
            at = slice(4096 * t, 4096 * t + x.shape[0])
            yz = (y[:, :, None] * z[:, None, :]).reshape(x.shape[0], -1).conj()
            back = lambda w: ((x.conj() @ w) * yz).sum(1)
            for b in range(3):
                B[b, at] = -c.facEwald * 4.0 * pi / L ** 3 * back(k[b] * eS).real
                if force:
                    for d in range(3):
                        F[d, at] -= c.facEwald * 8.0 * pi ** 2 / L ** 4 * mu[b, at] * back(k[b] * k[d] * eS).imag
        B += c.facEwald * (4.0 * self.al ** 3 / (3.0 * math.sqrt(pi)) * mu - 4.0 * pi / (3.0 * L ** 3) * mu.sum(1, keepdim=True))
        return B, F

    def interactions(self, mm, force=True):
        mu = mm * self.mag
        (b1, f1), (b2, f2) = self.pairs(mu, force), self.waves(mu, force)
        return b1 + b2, f1 + f2

    def normals(self):
        """Nine unit normals per particle: Philox4x32-10 of (particle, block, step) and Box-Muller."""
        M, i = 0xFFFFFFFF, torch.arange(self.n, dtype=torch.int64, device=DEV)
        z = []
        for b in range(3):
            w = [i, torch.full_like(i, b), torch.full_like(i, self.stepno & M), torch.full_like(i, self.stepno >> 32)]
            k0, k1 = self.seed & M, self.seed >> 32
            for _ in range(10):
                p, q = w[0] * 0xD2511F53, w[2] * 0xCD9E8D57
                w = [((q >> 32) & M) ^ w[1] ^ k0, q & M, ((p >> 32) & M) ^ w[3] ^ k1, p & M]
                k0, k1 = (k0 + 0x9E3779B9) & M, (k1 + 0xBB67AE85) & M
            u = [(v.double() + 0.5) * 2.0 ** -32 for v in w]
            for h in (0, 2):
                r = torch.sqrt(-2.0 * torch.log(u[h]))
                z += [r * torch.cos(2 * math.pi * u[h + 1]), r * torch.sin(2 * math.pi * u[h + 1])]
        return torch.stack(z[:9]).reshape(3, 3, self.n)

    def noise(self, dt):
        c, z = self.c, self.normals()
        kt = 2.0 * c.kB * c.temp / dt
        return (z[0] * torch.sqrt(kt * self.zr), z[1] * torch.sqrt(kt * c.magDamp / (c.gyroMr * c.satMag) / self.vol),
                z[2] * torch.sqrt(kt * self.zt))

    def slopes(self, m, e, B, torque, field):
        c = self.c
        dot = (m * e).sum(0)
        ext = torch.tensor([0.0, 0.0, c.magFluxDens if self.t < c.tMag else 0.0], dtype=torch.float64, device=DEV)[:, None]
        be = ext + B + c.anisConst * e * dot + field
        ke = (m - e * dot) * (self.v1 * dot) + torch.cross(torque, e, dim=0) * self.v2
        x = torch.cross(m, be, dim=0)
        return -c.velMmConst * (x + c.magDamp * torch.cross(m, x, dim=0)), ke

    def finish(self, m, e, force, dt):
        self.mm, self.ea = m / torch.linalg.norm(m, dim=0), e / torch.linalg.norm(e, dim=0)
        self.pos = _fold(self.pos + dt * force / self.zt, self.L)
        self.t += dt
        self.stepno += 1

    def step(self, dt):
        torque, field, fth = self.noise(dt)
        B, F = self.interactions(self.mm)
        k1, l1 = self.slopes(self.mm, self.ea, B, torque, field)
        m2, e2 = self.mm + dt * k1, self.ea + dt * l1
        k2, l2 = self.slopes(m2, e2, self.interactions(m2, False)[0], torque, field)
        self.finish(self.mm + dt / 2 * (k1 + k2), self.ea + dt / 2 * (l1 + l2), F + fth, dt)

    TABLEAUX = {
        0: ([[1.0]], [0.5, -0.5], [0.5, 0.5], 1 / 2),
        1: ([[1 / 2], [0, 3 / 4], [2 / 9, 1 / 3, 4 / 9]], [-5 / 72, 1 / 12, 1 / 9, -1 / 8], [2 / 9, 1 / 3, 4 / 9], 1 / 3),
        2: ([[1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9],
             [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
             [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656],
             [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]],
            [71 / 57600, 0, -71 / 16695, 71 / 1920, -17253 / 339200, 22 / 525, -1 / 40],
            [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84], 1 / 5),
    }

    def step_adaptive(self, dt):
        """One accepted step with the reference's step control; returns the next trial step."""
        c = self.c
        A, E, W, power = self.TABLEAUX[c.SOLVER]
        torque, field, fth = self.noise(dt)
        B, F = self.interactions(self.mm)
        failed = False
        total = lambda w, k: sum(a * b for a, b in zip(w, k) if a)
        while True:
            km, ke = [], []
            for s in range(len(E)):
                m = self.mm + dt * total(A[s - 1], km) if s else self.mm
                e = self.ea + dt * total(A[s - 1], ke) if s else self.ea
                if s:
                    B = self.interactions(m, False)[0]
                k, l = self.slopes(m, e, B, torque, field)
                km.append(k)
                ke.append(l)
            err = dt * float(torch.linalg.norm(total(E, km), dim=0).max())
            used = dt
            if err <= c.absTol:
                dt = dt if failed else dt * min(max(0.9 * (c.absTol / err) ** power, 0.2), 5.0)
                dt = max(dt, c.deltaTmin)
                break
            new = max(c.deltaTmin, dt * 0.5 if failed else dt * max(0.1, 0.9 * (c.absTol / err) ** power))
            torque, field = torque * math.sqrt(new / dt), field * math.sqrt(new / dt)
            dt, failed = new, True
        self.finish(self.mm + used * total(W, km), self.ea + used * total(W, ke), F + fth, used)
        return dt

    def state(self):
        return [x.cpu().numpy() for x in (self.pos, self.mm, self.ea)]


def _plain_rdf(s, case):
    """Pairs i < j < n - 1 and their distances, as the reference's analysis script counts them."""
    n, L = case["n"], s["sim"].lBox
    pos = torch.as_tensor(s["state"][0], device=DEV)
    r0 = 1e-8
    bw = 8.0 * r0 / case["bins"]
    count = torch.zeros(case["bins"], dtype=torch.int64, device=DEV)
    rows = max(1, int(2.5e7 // n))
    j = torch.arange(n, device=DEV)
    for a in range(0, n, rows):
        d = _fold(pos[:, None, :] - pos[:, a:a + rows, None], L)
        r2 = (d * d).sum(0)
        near = (r2 < (8.0 * r0) ** 2) & (j[None, :] > j[a:a + rows, None]) & (j[None, :] < n - 1)
        r = torch.sqrt(r2[near]).clamp(min=2 * r0)
        b = torch.floor(r * (1.0 / bw)).long()
        count += torch.bincount(b[b < case["bins"]], minlength=case["bins"])
    k = torch.arange(case["bins"], dtype=torch.float64, device=DEV) + 0.5
    return count.double() * (L ** 3 / (2 * s["cfg"].c.my_pi * bw ** 3 * n * n)) / k ** 2


def exact(case, seed):
    kind = case["kind"]
    if kind == "sweep":
        got = []
        for n, b, sd in _sweep_sizes(case, seed):
            s = _system(case, n, sd, b)
            p = _Plain(s, sd)
            s["sim"].close()
            for _ in range(case["steps"]):
                p.step(DT)
            got.append(p.state())
        return [np.concatenate([g[q] for g in got], axis=1) for q in range(3)]
    s = prepare(case, seed)
    if kind == "rdf":
        return [_plain_rdf(s, case).cpu().numpy(), None]
    p = _Plain(s, seed)
    if kind == "fields":
        B, F = p.interactions(p.mm)
        B2, _ = p.interactions(torch.as_tensor(s["other"], device=DEV), False)
        return [x.cpu().numpy() for x in (B, F, B2)]
    if kind == "adaptive":
        dt = DT
        for _ in range(case["steps"]):
            dt = p.step_adaptive(dt)
        return p.state() + [None, None]
    steps = case.get("steps", 1)
    if steps * case["n"] ** 2 > 4e10:
        return None
    for _ in range(steps):
        p.step(DT)
    return p.state()
