"""Pair forces, energy and virial with the type-pair table at one species,
several, and more than the default shared memory holds, with and without zero
pairs, against a brute-force FP64 sum."""
import math

import numpy as np
import pytest

from md_engine_b200 import Bounds, FixChargePairDSF, FixLJCut, FixLJCutFS, State, Vector

pytestmark = pytest.mark.gpu


# 55 and 64 species are the last whose table of four and of three floats a pair
# fits the default
@pytest.mark.parametrize("style", [FixLJCut, FixLJCutFS])
@pytest.mark.parametrize("ntypes,zero", [(1, False), (3, True), (60, False), (70, False)])
def test_forces_by_species(style, ntypes, zero):
    rng = np.random.default_rng(ntypes)
    n, L, rc = 1000, 11.0, 2.5
    g = np.stack(np.meshgrid(*[np.arange(10)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = ((g + 0.5) * 1.1 + rng.uniform(-0.1, 0.1, (n, 3))).astype(np.float32).astype(np.float64)
    types = rng.integers(0, ntypes, n)
    st = State()
    st.units.setLJ()
    st.bounds = Bounds(st, lo=Vector(0, 0, 0), hi=Vector(L, L, L))
    st.rCut, st.padding, st.dt = rc, 0.3, 0.001
    names = [f"T{k}" for k in range(ntypes)]
    for h in names:
        st.atomParams.addSpecies(h, 1.0, 1)
    st.addAtoms([names[t] for t in types], pos, np.zeros(n))
    sig = np.float32(1.0 - 0.1 * rng.random(ntypes)).astype(np.float64)
    eps = np.float32(0.5 + rng.random(ntypes)).astype(np.float64)
    if zero:
        eps[1] = 0.0
    fix = style(st, "pair")
    for k, h in enumerate(names):
        fix.setParameter("sig", h, h, sig[k])
        fix.setParameter("eps", h, h, eps[k])
    st.activateFix(fix)
    st.prepare()
    st.computeForces(1)
    f = st.getAtoms()[2]
    virial, energy = st.virials()[1], st.potentialEnergy()[0]
    d = pos[:, None] - pos[None]
    d -= L * np.round(d / L)
    r2 = (d ** 2).sum(2)
    np.fill_diagonal(r2, 1e9)
    s = np.sqrt(sig[:, None] * sig[None])[types][:, types]  # geometric mixing
    e = np.sqrt(eps[:, None] * eps[None])[types][:, types]

    def over_r(q2):
        s6 = s ** 6 / q2 ** 3
        return 24.0 * e * s6 * (2.0 * s6 - 1.0) / q2

    k = over_r(r2)
    if style is FixLJCutFS:
        k = k - over_r(rc * rc) * rc / np.sqrt(r2)
    ref = np.einsum("ij,ijc->ic", np.where(r2 < rc * rc, k, 0.0), d)
    rms = np.sqrt(np.mean(np.sum(ref ** 2, 1)))
    assert np.max(np.linalg.norm(f - ref, axis=1)) < 2e-4 * rms
    s6 = np.where(r2 < rc * rc, s ** 6 / r2 ** 3, 0.0)
    c6 = np.where(r2 < rc * rc, s ** 6 / rc ** 6, 0.0)
    u = 4.0 * e * (s6 * (s6 - 1.0) - c6 * (c6 - 1.0))
    if style is FixLJCutFS:
        u = u + np.where(r2 < rc * rc, over_r(rc * rc) * rc * (np.sqrt(r2) - rc), 0.0)
    w = np.where(r2 < rc * rc, k, 0.0)
    refv = 0.5 * np.array([np.sum(w * d[..., a] * d[..., b])
                           for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))])
    # FP32 separations are off by up to 2^-23 L = 1.3e-6, 1.6e-6 of the shortest
    # ones: 12 times that in r^-12, beside the terms' own rounding
    assert abs(energy - 0.5 * u.sum()) < 3e-5 * 0.5 * np.sum(4.0 * e * (s6 * (s6 + 1.0) + c6))
    assert np.max(np.abs(virial - refv)) < 3e-5 * 0.5 * np.sum(24.0 * e * s6 * (2.0 * s6 + 1.0))


def test_more_species_than_shared_memory_holds():
    n, ntypes = 150, 130
    st = State()
    st.units.setLJ()
    st.bounds = Bounds(st, lo=Vector(0, 0, 0), hi=Vector(20, 20, 20))
    st.rCut, st.padding, st.dt = 2.5, 0.3, 0.001
    names = [f"T{k}" for k in range(ntypes)]
    for h in names:
        st.atomParams.addSpecies(h, 1.0, 1)
    st.addAtoms([names[k % ntypes] for k in range(n)], np.random.default_rng(0).uniform(0, 20, (n, 3)), np.zeros(n))
    fix = FixLJCut(st, "pair")
    for h in names:
        fix.setParameter("sig", h, h, 0.1)
        fix.setParameter("eps", h, h, 1.0)
    st.activateFix(fix)
    with pytest.raises(RuntimeError, match="130 species"):
        st.prepare()


def test_charged_species_beyond_the_thirty_second():
    rng = np.random.default_rng(40)
    n, L, rc, alpha, ntypes = 1000, 11.0, 2.5, 0.4, 40
    g = np.stack(np.meshgrid(*[np.arange(10)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = ((g + 0.5) * 1.1 + rng.uniform(-0.1, 0.1, (n, 3))).astype(np.float32).astype(np.float64)
    types = rng.integers(32, ntypes, n)  # no atom of the first 32 species
    q = np.where(np.arange(n) % 2 == 0, 0.5, -0.5)
    st = State()
    st.units.setLJ()
    st.bounds = Bounds(st, lo=Vector(0, 0, 0), hi=Vector(L, L, L))
    st.rCut, st.padding, st.dt = rc, 0.3, 0.001
    names = [f"T{k}" for k in range(ntypes)]
    for h in names:
        st.atomParams.addSpecies(h, 1.0, 1)
    st.addAtoms([names[t] for t in types], pos, q)
    fix = FixLJCut(st, "pair")
    for h in names:
        fix.setParameter("sig", h, h, 1.0)
        fix.setParameter("eps", h, h, 1.0)
    st.activateFix(fix)
    dsf = FixChargePairDSF(st, "dsf")
    dsf.setParameters(alpha, rc)
    st.activateFix(dsf)
    st.prepare()
    st.computeForces()
    f = st.getAtoms()[2]
    d = pos[:, None] - pos[None]
    d -= L * np.round(d / L)
    r2 = (d ** 2).sum(2)
    np.fill_diagonal(r2, 1e9)
    r = np.sqrt(r2)
    erfc = np.vectorize(math.erfc)
    A = 2.0 * alpha / math.sqrt(math.pi)
    shift = math.erfc(alpha * rc) / rc ** 2 + A * math.exp(-(alpha * rc) ** 2) / rc
    near = r < rc
    lj = 24.0 * (2.0 / r2 ** 6 - 1.0 / r2 ** 3) / r2
    qq = q[:, None] * q[None]
    k = np.zeros_like(r)
    k[near] = lj[near] + qq[near] * (erfc(alpha * r[near]) / r2[near] + A * np.exp(-alpha ** 2 * r2[near]) / r[near]
                                     - shift) / r[near]
    ref = np.einsum("ij,ijc->ic", k, d)
    rms = np.sqrt(np.mean(np.sum(ref ** 2, 1)))
    assert np.max(np.linalg.norm(f - ref, axis=1)) < 2e-4 * rms
