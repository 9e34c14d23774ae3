"""What this library's speed is measured on: simulations and evaluations that
user programs run, through the Python front end, from the smallest boxes
(where launches and latency count) to the largest.

Every simulation case is one call of a program that drives the integrator with
its own arrays: positions and velocities in, a number of time steps,
positions, velocities and forces out, each call going on from the one before.

listed()   the cases            draw(rng)       one more of the same ranges
prepare()  inputs and handles   run()           one pass
work()     what a pass cannot do without
tolerance(), exact()            what its outputs are held to: exact() restates
    the physics in 64 bits with torch alone (brute-force pair sums, P3M by
    torch.fft, constraints by Newton iteration, energies differentiated by
    autograd)
"""
import math

import numpy as np
import torch

from md_engine_b200 import (BatchReplicas, Bounds, FixChargeEwald, FixChargePairDSF, FixLJCut, FixLJCutFS,
                            FixNoseHoover, FixPressureBerendsen, FixWCA, IntegratorVerlet, State, Vector, systems)

WATER_RC, WATER_SKIN, WATER_DT, WATER_TAU = 9.0, 1.0, 2.0, 100.0
REPLICA_SKIN = 0.8
ALPHA_RC = 2.7  # Ewald splitting parameter times the cutoff
FLUID_SKIN, FLUID_DT, FLUID_TAU = 0.3, 0.005, 0.5
SALT_RC = 3.0


def _interval(case):
    """turns between checks of the neighbour list: 10, or 5 where the box is
    too small for the molecule list and its margin"""
    return 5 if case["kind"] == "replicas" or (case["kind"] == "water" and case["n"] < 800) else 10


def listed():
    return [
        # Lennard-Jones fluid, NVT: a small box (every launch counts) ...
        {"name": "lj_4000", "kind": "lj", "n": 4000, "steps": 40, "style": "lj", "nvt": True},
        # ... the reference's benchmark size ...
        {"name": "lj_32000", "kind": "lj", "n": 32000, "steps": 20, "style": "lj", "nvt": True},
        # ... and a large one, energy-conserving
        {"name": "lj_256000", "kind": "lj", "n": 256000, "steps": 10, "style": "lj", "nvt": False},
        # charged Lennard-Jones particles (molten salt): Ewald sums without rigid molecules
        {"name": "salt_8000", "kind": "salt", "n": 8000, "steps": 20, "charge": "ewald"},
        # constant pressure: the box is rescaled during the run
        {"name": "npt_4000", "kind": "npt", "n": 4000, "steps": 20, "every": 10},
        # rigid TIP4P/2005 water, NVT, P3M: the smallest box of the examples' size class ...
        {"name": "water_512", "kind": "water", "n": 512, "steps": 20, "e3b": False},
        # ... the headline configuration, without and with the three-body term ...
        {"name": "water_4096", "kind": "water", "n": 4096, "steps": 20, "e3b": False},
        {"name": "water_e3b_4096", "kind": "water", "n": 4096, "steps": 20, "e3b": True},
        # ... and a box of about 100 A (128^3 mesh)
        {"name": "water_32768", "kind": "water", "n": 32768, "steps": 10, "e3b": False},
        # an ensemble of boxes of many sizes and temperatures advanced together
        {"name": "replicas_64", "kind": "replicas", "n": 64, "steps": 20, "e3b": True},
        # energies, pressure and forces of a stored frame (post-processing a trajectory)
        {"name": "frame_4096", "kind": "frame", "n": 4096},
        # one gradient of the three-body surrogate (training), host arrays
        {"name": "surrogate_4096", "kind": "surrogate", "n": 4096},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["lj", "lj", "salt", "npt", "water", "water", "water", "replicas", "frame", "surrogate"])
    if kind == "lj":
        return {"kind": kind, "n": size(1500, 200000), "steps": rng.choice([10, 20, 25]),
                "style": rng.choice(["lj", "wca", "ljfs"]), "nvt": rng.random() < 0.6}
    if kind == "salt":
        return {"kind": kind, "n": 2 * size(1000, 12000), "steps": 20, "charge": rng.choice(["ewald", "dsf"])}
    if kind == "npt":
        return {"kind": kind, "n": size(1500, 20000), "steps": 20, "every": rng.choice([5, 10])}
    if kind == "water":
        e3b = rng.random() < 0.5
        return {"kind": kind, "n": size(512, 8192 if e3b else 24000), "steps": rng.choice([10, 20]), "e3b": e3b}
    if kind == "replicas":
        return {"kind": kind, "n": size(4, 48), "steps": rng.choice([10, 20]), "e3b": rng.random() < 0.5}
    if kind == "frame":
        return {"kind": kind, "n": size(512, 12000)}
    return {"kind": kind, "n": 64 * size(4, 256)}


# ---- inputs -----------------------------------------------------------------
def _f32(a):
    """inputs that the library's 32-bit streams hold as they are"""
    return np.asarray(a, np.float64).astype(np.float32).astype(np.float64)


def _fluid_input(n, rho, T, seed, charged=False):
    """n particles at density rho near the sites of a face-centred (or, for a
    salt, simple cubic) lattice filled at random sites, Maxwell-Boltzmann
    velocities at T"""
    rng = np.random.default_rng(seed)
    base = np.array([[0, 0, 0]]) if charged else np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])
    k = int(math.ceil((n / len(base)) ** (1.0 / 3.0) - 1e-9))
    L = (n / rho) ** (1.0 / 3.0)
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)
    sites = (g[:, None, :] + base[None] + 0.25).reshape(-1, 3)
    parity = np.repeat(g.sum(1) % 2, len(base))
    if charged:  # as many of either sign, each on its own sublattice
        pick = np.concatenate([rng.permutation(np.flatnonzero(parity == p))[:n // 2] for p in (0, 1)])
        q = np.where(np.arange(n) < n // 2, 1.0, -1.0)
    else:
        pick = rng.permutation(len(sites))[:n]
        q = np.zeros(n)
    pos = sites[pick] * (L / k) + rng.normal(0.0, 0.05, (n, 3))
    vel = rng.standard_normal((n, 3)) * math.sqrt(T)
    vel -= vel.mean(0)
    return _f32(np.mod(pos, L)), _f32(vel), q, float(np.float32(L))


def _water_input(n, T, seed):
    s = systems.water_tip4p2005(nmol=n, T=T, seed=seed)
    s.pos, s.vel = _f32(s.pos), _f32(s.vel)
    return s


def _replica_inputs(case, seed):
    sizes, temps = systems.water_replica_sizes(case["n"], seed=20261203)
    return [(_water_input(int(m), float(T), seed + 7919 * k), float(T)) for k, (m, T) in enumerate(zip(sizes, temps))]


def _surrogate_input(case, seed):
    rng = np.random.default_rng(seed)
    w = np.concatenate([(rng.standard_normal(a * b) / math.sqrt(a)).tolist() + (0.1 * rng.standard_normal(b)).tolist()
                        for a, b in ((128, 64), (64, 64), (64, 64), (64, 16))]).astype(np.float32)
    x = rng.standard_normal((case["n"], 128)).astype(np.float32)
    t = rng.standard_normal((case["n"], 16)).astype(np.float32)
    return w, x, t


def _fluid_state(case, pos, vel, q, L, rc, T):
    st = State()
    st.units.setLJ()
    st.bounds = Bounds(st, lo=Vector(0, 0, 0), hi=Vector(L, L, L))
    st.rCut, st.padding, st.dt, st.periodicInterval = rc, FLUID_SKIN, FLUID_DT, _interval(case)
    st.atomParams.addSpecies(handle="A", mass=1.0, atomicNum=1)
    st.addAtoms(["A"] * len(pos), pos, q)
    st.setVelocities(np.arange(len(pos)), vel)
    if T is not None:
        nh = FixNoseHoover(st, "nvt", "all")
        nh.setTemperature(T, FLUID_TAU)
        st.activateFix(nh)
    return st


def _water_state(case, s, T, e3b, skin=WATER_SKIN):
    return systems.build_water_state(s, rcut=WATER_RC, skin=skin, dt=WATER_DT, interval=_interval(case),
                                     grid=_mesh(s.L[0]), e3b=e3b, T=T, tau=WATER_TAU, alpha=ALPHA_RC / WATER_RC)


def _mesh(L):
    return max(32, systems.p3m_mesh_for(L))


class _Program:
    """what a user's program holds between its calls"""


def prepare(case, seed):
    p = _Program()
    p.case = case
    kind = case["kind"]
    if kind in ("lj", "npt", "salt"):
        T, rho, rc = _fluid_conditions(case)
        pos, vel, q, L = _fluid_input(case["n"], rho, T, seed, kind == "salt")
        p.state = _fluid_state(case, pos, vel, q, L, rc, T if case.get("nvt", True) else None)
        fix = {"wca": FixWCA, "ljfs": FixLJCutFS}.get(case.get("style"), FixLJCut)(p.state, "pair")
        fix.setParameter("sig", "A", "A", 1.0)
        fix.setParameter("eps", "A", "A", 1.0)
        p.state.activateFix(fix)
        if kind == "salt":
            if case["charge"] == "ewald":
                c = FixChargeEwald(p.state, "charge", "all")
                c.setParameters(_mesh(L), _mesh(L), _mesh(L), rc, 5)
                c.setAlpha(ALPHA_RC / rc)
            else:
                c = FixChargePairDSF(p.state, "charge", "all")
                c.setParameters(0.25, rc)
            p.state.activateFix(c)
        if kind == "npt":
            p.barostat = FixPressureBerendsen(p.state, "npt", 1.0, 1.0, case["every"])
            p.state.activateFix(p.barostat)
    elif kind == "water":
        p.state, _ = _water_state(case, _water_input(case["n"], 298.0, seed), 298.0, case["e3b"])
    elif kind == "frame":
        p.state, _ = _water_state(case, _water_input(case["n"], 298.0, seed), 298.0, True)
        p.frame = _water_input(case["n"], 298.0, seed + 1).pos  # the stored frame
    elif kind == "replicas":
        p.states = []
        for s, T in _replica_inputs(case, seed):
            st, _ = _water_state(case, s, T, case["e3b"], skin=REPLICA_SKIN)
            st.nThreadPerAtom = 32
            p.states.append(st)
        p.batch = BatchReplicas(p.states)
        p.batch.prepare()
        return p
    else:
        w, p.x, p.t = _surrogate_input(case, seed)
        p.state, fixes = _water_state(case, _water_input(512, 298.0, seed), 298.0, True)
        p.state.prepare()
        p.e3b = fixes["e3b"]
        p.e3b.surrogateSetParams(w, np.zeros(128, np.float32), np.ones(128, np.float32), 1.0)
        return p
    p.state.prepare()
    p.integrator = IntegratorVerlet(p.state)
    p.x, p.v, _ = p.state.getAtoms()
    return p


def run(p):
    case = p.case
    kind = case["kind"]
    if kind in ("lj", "salt", "water"):
        out = p.integrator.runHost(case["steps"], p.x, p.v)
        p.x, p.v = out["pos"], out["vel"]
        return out["pos"], out["vel"], out["force"]
    if kind == "npt":
        p.integrator.run(case["steps"])
        x, v, f = p.state.getAtoms()
        return x, v, f, p.state.bounds.hi.v - p.state.bounds.lo.v, p.barostat.lastPressure
    if kind == "replicas":
        p.batch.run(case["steps"])
        atoms = [st.getAtoms() for st in p.states]
        return tuple(np.concatenate([a[k] for a in atoms]) for k in range(3))
    if kind == "frame":
        p.state.putAtoms(positions=p.frame)
        p.state.buildNeighborlists()
        p.state.computeForces()
        energies = p.state.potentialEnergy()
        pressure, virial = p.state.pressure()
        return p.state.getAtoms()[2], energies, pressure, virial
    loss, grad = p.e3b.surrogateGrad(p.x, p.t)
    return loss, grad


def _fluid_conditions(case):
    """temperature, density, cutoff"""
    if case["kind"] == "salt":
        return 1.5, 0.6, SALT_RC
    return 1.2, 0.8442, 2.5


# ---- what a pass cannot do without ------------------------------------------
def work(case):
    kind, n = case["kind"], case["n"]
    if kind == "surrogate":
        macs = 128 * 64 + 2 * 64 * 64 + 64 * 16
        return {"bytes": 4 * n * (128 + 16) + 8 * 17616, "flops": 3 * 2 * macs * n}
    if kind in ("lj", "npt", "salt"):
        T, rho, rc = _fluid_conditions(case)
        rc = 2.0 ** (1.0 / 6.0) if case.get("style") == "wca" else rc
        per = rho * 2.0 / 3.0 * math.pi * rc ** 3 * (60 if kind == "salt" else 30)  # each pair once
        # per step: positions, velocities and forces in and out (float4)
        return {"bytes": case["steps"] * n * 96, "flops": case["steps"] * n * per}
    mols = int(systems.water_replica_sizes(n, seed=20261203)[0].sum()) if kind == "replicas" else n
    e3b = case.get("e3b", True)
    steps = case.get("steps", 2)
    pairs = 0.0333 * 2.0 / 3.0 * math.pi * WATER_RC ** 3  # molecule pairs per molecule, each once
    mesh = 30.0 * 64 * 1.2  # mesh points per molecule (1.2 points per A^3) times 4 transforms
    flops = mols * (pairs * (9 * 45 + 15) + 3 * 125 * 10 + mesh * 5 + (40 * 150 if e3b else 0))
    return {"bytes": steps * mols * 4 * 96, "flops": steps * flops}


# ---- tolerance --------------------------------------------------------------
# About four times what two correct 32-bit runs differ by: the mesh charges are
# summed by atomics in any order, and three passes on, the trajectories of two
# runs of one program are 1e-5 to 5e-5 apart (velocities, forces; 4e-3 of the
# root mean square at the worst atom); a run is 2e-5 to 7e-5 from exact() after
# its first pass.  A frame's sums are 5e-6 from exact(), a gradient of the
# surrogate's 16-bit layers 2e-3 to 3e-3.
def tolerance(case):
    kind = case["kind"]
    if kind == "surrogate":
        return {"rel": 1e-2, "max": 0.1}
    if kind == "frame":
        return {"rel": 2e-5, "max": 1e-3}
    return {"rel": 2e-4, "max": 2e-2}


# ---- the same in 64 bits ----------------------------------------------------
DEV = torch.device("cuda" if torch.cuda.is_available() else "cpu")
REAL = {"boltz": 0.0019872067, "mvv": 48.88821291 ** 2, "qqr": 332.06371, "press": 68568.415}
LJ = {"boltz": 1.0, "mvv": 1.0, "qqr": 1.0, "press": 1.0}


def _t(a):
    return torch.as_tensor(np.asarray(a), dtype=torch.float64, device=DEV)


def _image(d, L):
    return d - L * torch.round(d / L)


def _pair_sum(x, L, rc, term):
    """forces, energy and virial (xx yy zz xy xz yz) of a pair term over all
    pairs within rc: term(i, j, r2) gives F = s (x_i - x_j) and the energy of
    each pair; rows in slabs along x, so that far columns are left out"""
    n = len(x)
    xw, order = torch.sort(torch.remainder(x[:, 0], L))
    ext = torch.cat([xw - L, xw, xw + L])
    f = torch.zeros_like(x)
    e = torch.zeros((), dtype=torch.float64, device=x.device)
    w = torch.zeros(6, dtype=torch.float64, device=x.device)
    rows = max(1, min(1024, int(2e7) // n + 64))
    for a in range(0, n, rows):
        b = min(n, a + rows)
        lo = int(torch.searchsorted(ext, xw[a] - rc))
        hi = int(torch.searchsorted(ext, xw[b - 1] + rc, right=True))
        cols = torch.arange(lo, hi, device=x.device) % n if hi - lo < n else torch.arange(n, device=x.device)
        i, j = order[a:b], order[cols]
        d = [_image(x[i, c][:, None] - x[j, c][None, :], L) for c in range(3)]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        off = (r2 >= rc * rc) | (i[:, None] == j[None, :])
        r2.masked_fill_(off, rc * rc)
        s, u = term(i, j, r2)
        s.masked_fill_(off, 0.0)
        for c in range(3):
            f[i, c] += (s * d[c]).sum(1)
        e += 0.5 * u.masked_fill(off, 0.0).sum()
        for c, (p, q) in enumerate(((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))):
            w[c] += 0.5 * (s * d[p] * d[q]).sum()
    return f, e, w


def _lj_term(eps, sig, rc, style="lj"):
    def force_over_r(r2):
        s6 = sig ** 6 / r2 ** 3
        return 24.0 * eps * s6 * (2.0 * s6 - 1.0) / r2

    shift = (sig / rc) ** 12 - (sig / rc) ** 6
    f_rc = force_over_r(rc * rc) * rc

    def term(i, j, r2):
        s = force_over_r(r2)
        if style == "ljfs":
            s = s - f_rc / torch.sqrt(r2)
        s6 = sig ** 6 / r2 ** 3
        return s, 4.0 * eps * (s6 * (s6 - 1.0) - shift)
    return term


def _ewald_term(q, mol, alpha, qqr):
    """real space; pairs inside a molecule carry the exclusion correction"""
    def term(i, j, r2):
        r = torch.sqrt(r2)
        qq = qqr * q[i][:, None] * q[j][None, :]
        own = mol[i][:, None] == mol[j][None, :] if mol is not None else torch.zeros_like(r2, dtype=torch.bool)
        u = (torch.erfc(alpha * r) - own.double()) / r
        s = (u + 2.0 * alpha / math.sqrt(math.pi) * torch.exp(-alpha * alpha * r2)) / r2
        return qq * s, qq * u
    return term


def _dsf_term(q, alpha, rc):
    A = 2.0 * alpha / math.sqrt(math.pi)
    shift = math.erfc(alpha * rc) / rc ** 2 + A * math.exp(-(alpha * rc) ** 2) / rc

    def term(i, j, r2):
        r = torch.sqrt(r2)
        qq = q[i][:, None] * q[j][None, :]
        s = (torch.erfc(alpha * r) / r2 + A * torch.exp(-alpha * alpha * r2) / r - shift) / r
        return qq * s, torch.zeros_like(s)
    return term


class _P3M:
    """order-5 particle-particle particle-mesh sum on an n^3 mesh"""

    def __init__(self, L, n, alpha, qqr):
        self.L, self.n, self.alpha, self.qqr = L, n, alpha, qqr
        h = L / n
        k1 = 2.0 * math.pi / L * torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device=DEV)
        self.k = [k1.reshape([-1 if c == d else 1 for c in range(3)]) for d in range(3)]
        lim = int(alpha * h / 3.14159 * math.sqrt(-math.log(10e-7))) + 1
        self.k2 = sum(k * k for k in self.k)
        s1, s2 = torch.zeros_like(self.k2), torch.zeros_like(self.k2)
        steps = range(-lim, lim + 1)
        for mx in steps:
            for my in steps:
                for mz in steps:
                    m = [k + 2.0 * math.pi / h * a for k, a in zip(self.k, (mx, my, mz))]
                    mm = sum(a * a for a in m)
                    W = torch.ones(1, dtype=torch.float64, device=DEV)
                    for a in m:
                        W = W * torch.sinc(a * h / (2.0 * math.pi)) ** 10
                    dot = sum(k * a for k, a in zip(self.k, m))
                    s1 += 4.0 * math.pi * torch.exp(-mm / (4.0 * alpha ** 2)) * dot / mm.clamp_min(1e-300) * W
                    s2 += W
        self.G = torch.where(self.k2 > 0, s1 / s2 ** 2 / self.k2.clamp_min(1e-300), 0.0)

    def _stencil(self, x):
        h = self.L / self.n
        at = torch.floor(x / h + 0.5)
        u = x / h - at
        u2, u4 = u * u, u ** 4
        w = torch.stack([(1 - 8 * u + 24 * u2 - 32 * u * u2 + 16 * u4) / 384,
                         (19 - 44 * u + 24 * u2 + 16 * u * u2 - 16 * u4) / 96,
                         (115 - 120 * u2 + 48 * u4) / 192,
                         (19 + 44 * u + 24 * u2 - 16 * u * u2 - 16 * u4) / 96,
                         (1 + 8 * u + 24 * u2 + 32 * u * u2 + 16 * u4) / 384])
        p = torch.stack([torch.remainder(at.long() + c, self.n) for c in range(-2, 3)])
        for a in range(5):
            for b in range(5):
                for c in range(5):
                    yield ((p[a, :, 0] * self.n + p[b, :, 1]) * self.n + p[c, :, 2],
                           w[a, :, 0] * w[b, :, 1] * w[c, :, 2])

    def __call__(self, x, q):
        n, V = self.n, self.L ** 3
        qs = q * math.sqrt(self.qqr)
        rho = torch.zeros(n ** 3, dtype=torch.float64, device=DEV)
        for cell, w in self._stencil(x):
            rho.index_add_(0, cell, w * qs)
        rk = torch.fft.fftn(rho.reshape(n, n, n))
        field = [-torch.fft.ifftn(1j * k * rk * self.G).real.reshape(-1) * n ** 3 / V for k in self.k]
        f = torch.zeros_like(x)
        for cell, w in self._stencil(x):
            for c in range(3):
                f[:, c] += w * field[c][cell]
        f *= qs[:, None]
        E = self.G * (rk.real ** 2 + rk.imag ** 2)
        energy = 0.5 / V * E.sum() - self.alpha / math.sqrt(math.pi) * (qs * qs).sum()
        d = torch.where(self.k2 > 0, -2.0 * (1.0 / self.k2.clamp_min(1e-300) + 0.25 / self.alpha ** 2), 0.0)
        vir = [0.5 / V * ((float(a == b) + d * self.k[a] * self.k[b]) * E).sum()
               for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))]
        return f, energy, torch.stack(vir)


def _e3b(x, L):
    """E3B3 three-body water (sites O, H1, H2, M per molecule): forces by
    autograd, [two-body, three-body] energies, virial as sum_i x_i F_i over
    relative positions of each pair term"""
    kj = 0.23900573614
    E2, Ea, Eb, Ec = 453000.0 * kj, 150.0 * kj, -1005.0 * kj, 1880.0 * kj
    k2, k3, rs, rf, rlist, rmax = 4.872, 1.907, 5.0, 5.2, 6.2, 6.1572
    O = x[0::4]
    near_i, near_j = [], []
    for a in range(0, len(O), 512):
        d = _image(O[a:a + 512, None, :] - O[None], L)
        r2 = (d * d).sum(2)
        i, j = torch.nonzero((r2 < rlist ** 2) & (r2 > 0), as_tuple=True)
        near_i.append(i + a)
        near_j.append(j)
    i, j = torch.cat(near_i), torch.cat(near_j)
    sep = [_image(O[i] - O[j], L)]
    sep += [_image(x[h::4][j] - O[i], L) for h in (1, 2)]  # H of j from O of i
    sep = [s.detach().requires_grad_(True) for s in sep]
    with torch.enable_grad():
        r = torch.linalg.norm(sep[0], dim=1)
        two = 0.5 * (E2 * torch.exp(-k2 * r)).sum()
        inside = (r <= rmax).double()

        def e(d):
            rr = torch.linalg.norm(d, dim=1)
            sw = (rf - rr) ** 2 * (rf + 2 * rr - 3 * rs) / (rf - rs) ** 3
            sw = torch.where(rr <= rs, torch.ones_like(rr), torch.where(rr > rf, torch.zeros_like(rr), sw))
            return inside * sw * torch.exp(-k3 * rr)

        pb, pc = e(sep[1]), e(sep[2])
        # the reversed pair (j, i) of every ordered pair (i, j)
        key, rkey = i * len(O) + j, j * len(O) + i
        back = torch.argsort(key)[torch.searchsorted(torch.sort(key)[0], rkey)]
        s = pb + pc
        rev = s[back]
        zero = torch.zeros(len(O), dtype=torch.float64, device=x.device)
        Tx = zero.index_add(0, i, s)
        Ty, Tz = zero.index_add(0, j, pb), zero.index_add(0, j, pc)
        three = 0.5 * (Ea * ((Ty[j] - pb) * pc + (Tz[j] - pc) * pb) + Eb * (Tx[j] + Ty[i] + Tz[i] - 2 * rev) * s +
                       Ec * (Tx[i] - s) * s).sum()
        grads = torch.autograd.grad(two + three, sep)
    f = torch.zeros_like(x)
    f[0::4].index_add_(0, i, -grads[0])
    f[0::4].index_add_(0, j, grads[0])
    vir = torch.zeros(6, dtype=torch.float64, device=x.device)
    for h in (1, 2):
        f[h::4].index_add_(0, j, -grads[h])
        f[0::4].index_add_(0, i, grads[h])
    for c, (a, b) in enumerate(((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))):
        vir[c] = sum((-g[:, a] * d[:, b].detach()).sum() for g, d in zip(grads, sep))
    return f, torch.stack([two.detach(), three.detach()]), vir


class _Fluid:
    units, molecules = LJ, False

    def __init__(self, case, L, q, style):
        self.case, self.L, self.q, self.style = case, L, _t(q), style
        _, _, self.rc = _fluid_conditions(case)
        self.skin, self.dt, self.tau = FLUID_SKIN, FLUID_DT, FLUID_TAU
        self.p3m = _P3M(L, _mesh(L), ALPHA_RC / self.rc, 1.0) if case.get("charge") == "ewald" else None
        n = case["n"]
        self.mass, self.ndf = torch.ones(n, dtype=torch.float64, device=DEV), 3 * n

    def evaluate(self, x):
        rc = 2.0 ** (1.0 / 6.0) if self.style == "wca" else self.rc
        f, e, w = _pair_sum(x, self.L, rc, _lj_term(1.0, 1.0, rc, self.style))
        if self.case["kind"] == "salt":
            alpha = ALPHA_RC / self.rc
            term = _ewald_term(self.q, None, alpha, 1.0) if self.p3m else _dsf_term(self.q, 0.25, self.rc)
            f = f + _pair_sum(x, self.L, self.rc, term)[0]
            if self.p3m:
                f = f + self.p3m(x, self.q)[0]
        return f, None, w


class _Water:
    units, molecules = REAL, True
    r_OH, r_HH, r_OM, gamma = 0.9572, 1.5139, 0.1546, 0.73612446364836

    def __init__(self, n, L, e3b, skin):
        self.L, self.e3b, self.skin, self.dt, self.tau = L, e3b, skin, WATER_DT, WATER_TAU
        self.alpha = ALPHA_RC / WATER_RC
        self.p3m = _P3M(L, _mesh(L), self.alpha, REAL["qqr"])
        q = _t([systems.QH, systems.QH, systems.QM]).float().double()
        self.qc = q.repeat(n)
        self.mol = torch.arange(n, device=DEV).repeat_interleave(3)
        m = _t([systems.MASS_O, systems.MASS_H, systems.MASS_H, 0.0])
        self.mass, self.ndf = m.repeat(n), 6 * n

    def evaluate(self, x):
        f = torch.zeros_like(x)
        O, charged = x[0::4], x.reshape(-1, 4, 3)[:, 1:].reshape(-1, 3)
        fo, elj, w = _pair_sum(O, self.L, WATER_RC, _lj_term(systems.EPS_OO, systems.SIG_OO, WATER_RC))
        f[0::4] += fo
        fr, er, wr = _pair_sum(charged, self.L, WATER_RC, _ewald_term(self.qc, self.mol, self.alpha, REAL["qqr"]))
        fk, ek, wk = self.p3m(charged, self.qc)
        f.reshape(-1, 4, 3)[:, 1:] += (fr + fk).reshape(-1, 3, 3)
        e3, w = torch.zeros(2, dtype=torch.float64, device=DEV), w + wr + wk
        if self.e3b:
            f3, e3, w3 = _e3b(x, self.L)
            f, w = f + f3, w + w3
        return f, torch.cat([torch.stack([elj + er, ek]), e3]), w

    # rigid molecules: sites O, H1, H2, M
    def whole(self, x):
        m = x.reshape(-1, 4, 3)
        return (m[:, :1] + _image(m - m[:, :1], self.L)).reshape(-1, 3)

    def place_m(self, x):
        m = x.reshape(-1, 4, 3)
        s = m[:, 1] + m[:, 2] - 2.0 * m[:, 0]
        m[:, 3] = m[:, 0] + self.r_OM * s / torch.linalg.norm(s, dim=1, keepdim=True)
        return x

    def _bonds(self, a):
        a = a.reshape(-1, 4, 3)
        return torch.stack([a[:, 0] - a[:, 1], a[:, 0] - a[:, 2], a[:, 1] - a[:, 2]], 1)

    def _push(self, g, r):
        """displacements of O, H1, H2 under multipliers g along bonds r, over the masses"""
        c = g[:, :, None] * r
        d = torch.zeros(len(g), 4, 3, dtype=torch.float64, device=DEV)
        d[:, 0] = (c[:, 0] + c[:, 1]) / systems.MASS_O
        d[:, 1] = (-c[:, 0] + c[:, 2]) / systems.MASS_H
        d[:, 2] = (-c[:, 1] - c[:, 2]) / systems.MASS_H
        return d

    def constrain_x(self, x0, x, v):
        """positions x (moved from x0 unconstrained) back onto the rigid
        geometry by forces along the bonds of x0; velocities follow"""
        r0 = self._bonds(self.whole(x0))
        x = self.whole(x)
        length2 = _t([self.r_OH ** 2, self.r_OH ** 2, self.r_HH ** 2])
        g = torch.zeros(len(r0), 3, dtype=torch.float64, device=DEV)
        unit = torch.eye(3, dtype=torch.float64, device=DEV)
        cols = [self._bonds(self._push(unit[k].expand(len(r0), 3), r0)) for k in range(3)]
        for _ in range(8):
            b = self._bonds(x) + self._bonds(self._push(g, r0))
            c = (b * b).sum(2) - length2
            J = torch.stack([2.0 * (b * cols[k]).sum(2) for k in range(3)], 2)
            g = g - torch.linalg.solve(J, c[:, :, None])[:, :, 0]
        d = self._push(g, r0).reshape(-1, 3)
        return x + d, v + d / self.dt

    def constrain_v(self, x, v):
        r = self._bonds(self.whole(x))
        unit = torch.eye(3, dtype=torch.float64, device=DEV)
        J = torch.stack([(r * self._bonds(self._push(unit[k].expand(len(r), 3), r))).sum(2) for k in range(3)], 2)
        c = (r * self._bonds(v)).sum(2)
        g = -torch.linalg.solve(J, c[:, :, None])[:, :, 0]
        return v + self._push(g, r).reshape(-1, 3)

    def share_m(self, f):
        m = f.reshape(-1, 4, 3).clone()
        m[:, 0] += self.gamma * m[:, 3]
        m[:, 1] += 0.5 * (1.0 - self.gamma) * m[:, 3]
        m[:, 2] += 0.5 * (1.0 - self.gamma) * m[:, 3]
        m[:, 3] = 0.0
        return m.reshape(-1, 3)


class _Chain:
    """Nose-Hoover chain of ten thermostats, one half step at a time"""

    def __init__(self, ke, ndf, kT, tau, dt):
        self.ke, self.nkt, self.kT, self.dt = ke, ndf * kT, kT, dt
        self.m = [ndf * kT * tau * tau] + [kT * tau * tau] * 9
        self.v = [0.0] * 10
        self.f = [(ke - self.nkt) / self.m[0]] + [-kT / self.m[1]] * 9

    def half(self, ke=None):
        if ke is not None:
            self.ke = ke
            self.f[0] = (ke - self.nkt) / self.m[0]
        v, f, dt = self.v, self.f, self.dt
        v[9] += 0.25 * dt * f[9]
        for k in range(8, -1, -1):
            s = math.exp(-0.125 * dt * v[k + 1])
            v[k] = (v[k] * s + 0.25 * dt * f[k]) * s
        scale = math.exp(-0.5 * dt * v[0])
        self.ke *= scale * scale
        for k in range(9):
            s = math.exp(-0.125 * dt * v[k + 1])
            f[k] = (self.ke - self.nkt) / self.m[0] if k == 0 else \
                (self.m[k - 1] * v[k - 1] ** 2 - self.kT) / self.m[k]
            v[k] = (v[k] * s + 0.25 * dt * f[k]) * s
        f[9] = (self.m[8] * v[8] ** 2 - self.kT) / self.m[9]
        v[9] += 0.25 * dt * f[9]
        return scale


def _wrap(sys_, x):
    if not sys_.molecules:
        return torch.remainder(x, sys_.L)
    m = x.reshape(-1, 4, 3)
    return (m - sys_.L * torch.floor(m[:, :1] / sys_.L)).reshape(-1, 3)


def _simulate(sys_, x, v, T, steps, interval, every=0):
    """velocity Verlet from x, v with the library's order of operations; the
    Berendsen barostat (pressure 1, time 1, bulk modulus 10, dilation within
    1e-5) acts after the step of every turn that is a multiple of `every`"""
    u, dt = sys_.units, sys_.dt
    real = sys_.mass > 0
    kick = torch.where(real, 0.5 * dt / u["mvv"] / sys_.mass.clamp_min(1e-300), torch.zeros_like(sys_.mass))[:, None]
    lo = 0.0

    def ke():
        return float((sys_.mass[:, None] * v * v).sum()) * u["mvv"]

    x = _wrap(sys_, sys_.whole(x) if sys_.molecules else x)
    f = sys_.evaluate(x)[0]
    last = x.clone()
    if sys_.molecules:
        x, v = sys_.constrain_x(x, x, v)
        x, v = sys_.place_m(x), sys_.constrain_v(x, v)
        v = v - (sys_.mass[:, None] * v).sum(0) / sys_.mass.sum()
    chain = _Chain(ke(), sys_.ndf, u["boltz"] * T, sys_.tau, dt) if T is not None else None
    scale = chain.half() if chain else 1.0
    final = 1.0
    pressure = None
    for k in range(steps):
        if k % interval == 0 and bool(((_image(x - last, sys_.L) ** 2).sum(1) > 0.25 * sys_.skin ** 2).any()):
            x = _wrap(sys_, x - lo) + lo
            last = x.clone()
        v = torch.where(real[:, None], v * scale + kick * f, 0.0)
        x0, x = x, x + dt * v
        if sys_.molecules:
            x, v = sys_.constrain_x(x0, x, v)
            x, v = sys_.place_m(x), torch.where(real[:, None], v, 0.0)
        f, _, w = sys_.evaluate(x)
        f = sys_.share_m(f) if sys_.molecules else f
        v = v + kick * f
        if sys_.molecules:
            v = sys_.constrain_v(x, v)
        if chain:
            final = chain.half(ke())
            scale = final * chain.half()
        if every and k % every == 0:
            pressure = (ke() + float(w[:3].sum())) / (3.0 * sys_.L ** 3) * u["press"]
            s = (1.0 - dt * (1.0 - pressure) / 10.0) ** (1.0 / 3.0)
            s = min(max(s, 1.0 - 1e-5), 1.0 + 1e-5)
            c = lo + 0.5 * sys_.L
            x = c + (x - c) * s
            sys_.L *= s
            lo = c - 0.5 * sys_.L
            x = _wrap(sys_, x - lo) + lo
            last = x.clone()
    return x, v * final, f, pressure


def _surrogate_exact(case, seed):
    w, x, t = _surrogate_input(case, seed)
    w, x, t = _t(w).requires_grad_(True), _t(x), _t(t)
    with torch.enable_grad():
        at, a = 0, x
        for layer, (n, m) in enumerate(((128, 64), (64, 64), (64, 64), (64, 16))):
            a = a @ w[at:at + n * m].reshape(n, m) + w[at + n * m:at + n * m + m]
            a = torch.nn.functional.silu(a) if layer < 3 else a
            at += n * m + m
        loss = ((a - t)[:, :9] ** 2).mean()
        (g,) = torch.autograd.grad(loss, w)
    return float(loss.detach()), g.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "surrogate":
        return _surrogate_exact(case, seed)
    if kind in ("lj", "salt", "npt"):
        T, rho, _ = _fluid_conditions(case)
        pos, vel, q, L = _fluid_input(case["n"], rho, T, seed, kind == "salt")
        s = _Fluid(case, L, q, case.get("style", "lj"))
        x, v, f, p = _simulate(s, _t(pos), _t(vel), T if case.get("nvt", True) else None, case["steps"],
                               _interval(case), case.get("every", 0))
        out = tuple(a.cpu().numpy() for a in (x, v, f))
        return out + (np.full(3, s.L), p) if kind == "npt" else out
    if kind == "water":
        w = _water_input(case["n"], 298.0, seed)
        s = _Water(case["n"], float(w.L[0]), case["e3b"], WATER_SKIN)
        xvf = _simulate(s, _t(w.pos), _t(w.vel), 298.0, case["steps"], _interval(case))[:3]
        return tuple(a.cpu().numpy() for a in xvf)
    if kind == "replicas":
        outs = []
        for w, T in _replica_inputs(case, seed):
            s = _Water(len(w.molecules), float(w.L[0]), case["e3b"], REPLICA_SKIN)
            xvf = _simulate(s, _t(w.pos), _t(w.vel), T, case["steps"], _interval(case))[:3]
            outs.append([a.cpu().numpy() for a in xvf])
        return tuple(np.concatenate([o[k] for o in outs]) for k in range(3))
    first, frame = _water_input(case["n"], 298.0, seed), _water_input(case["n"], 298.0, seed + 1)
    s = _Water(case["n"], float(frame.L[0]), True, WATER_SKIN)
    x, v = _t(first.pos), _t(first.vel)
    x, v = s.constrain_x(x, x, v)
    v = s.constrain_v(x, v)
    v = v - (s.mass[:, None] * v).sum(0) / s.mass.sum()
    f, e, w = s.evaluate(_t(frame.pos))
    ke = float((s.mass[:, None] * v * v).sum()) * REAL["mvv"]
    pressure = (ke + float(w[:3].sum())) / (3.0 * s.L ** 3) * REAL["press"]
    return f.cpu().numpy(), e.cpu().numpy(), pressure, w.cpu().numpy()
