"""Observables' device sums around their block size, against the sums of the
per-atom values they add."""
import numpy as np
import pytest

from md_engine_b200 import Bounds, FixLJCut, State, Vector

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 255, 256, 257, 4097])
def test_virial_energy_and_kinetic_sums(oracle, n):
    rng = np.random.default_rng(n)
    L = max(9.0, (n / 0.4) ** (1 / 3))
    k = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    st = State()
    st.units.setLJ()
    st.bounds = Bounds(st, lo=Vector(0, 0, 0), hi=Vector(L, L, L))
    st.rCut, st.padding, st.dt = 2.5, 0.3, 0.001
    st.atomParams.addSpecies("A", 2.0, 1)
    st.addAtoms(["A"] * n, (g + 0.5) * min(L / k, 1.3) + rng.uniform(-0.1, 0.1, (n, 3)), np.zeros(n))
    v = rng.standard_normal((n, 3)).astype(np.float32).astype(np.float64)
    st.setVelocities(np.arange(n), v)
    lj = FixLJCut(st, "lj")
    lj.setParameter("sig", "A", "A", 1.0)
    lj.setParameter("eps", "A", "A", 1.0)
    st.activateFix(lj)
    st.prepare()
    p, w = st.pressure()
    per, total = st.virials()
    # the same FP32 terms added in FP64: only the order of the additions differs
    size = np.abs(per).sum(0)
    assert np.all(np.abs(total - per.sum(0)) <= 1e-13 * size) and np.all(np.abs(w - per.sum(0)) <= 1e-13 * size)
    mv2, _ = st.kinetic()
    assert abs(mv2 - 2.0 * np.sum(v ** 2)) < 1e-7 * mv2  # 1/m is FP32
    assert abs(p - (mv2 + w[:3].sum()) / (3.0 * L ** 3)) < 1e-9 * (mv2 + size[:3].sum()) / L ** 3
    x = st.getAtoms()[0]
    c, nb, _ = st.getNeighborList()
    prm = oracle.lj_params(1, {(0, 0): 1.0}, {(0, 0): 1.0}, 2.5)
    ref = oracle.pair_forces(x, np.zeros(n, int), np.zeros(n), prm, np.full(3, L), c, nb, want=("energy",))
    assert abs(st.potentialEnergy()[0] - ref["energy"].sum()) < 1e-5 * np.abs(ref["energy"]).sum()
