"""The end of a fused step (kinetic sum over the second half's blocks, the
Nose-Hoover chain) on an ideal gas, whose velocities only the chain changes:
against the FP64 chain, at block counts with one, two and more partial sums per
thread, inside and outside the range of the polynomial exponential."""
import numpy as np
import pytest

from md_engine_b200 import Bounds, FixLJCut, FixNoseHoover, IntegratorVerlet, State, Vector

pytestmark = pytest.mark.gpu


# (with a 0.01 tau the FP64 chain itself overflows from a few thousand atoms on)
@pytest.mark.parametrize("n,tau", [(1, 0.5), (256, 0.5), (257, 0.5), (66049, 0.5), (1, 0.01), (256, 0.01), (257, 0.01)])
def test_chain_scales_an_ideal_gas(oracle, n, tau):
    rng = np.random.default_rng(n)
    L, dt, T, steps = 60.0, 0.005, 1.0, 7
    v0 = np.asarray(rng.standard_normal((n, 3)) * np.sqrt(3.0 * T), np.float32).astype(np.float64)
    st = State()
    st.units.setLJ()
    st.bounds = Bounds(st, lo=Vector(0, 0, 0), hi=Vector(L, L, L))
    st.rCut, st.padding, st.dt, st.periodicInterval = 1.0, 0.5, dt, 5
    st.atomParams.addSpecies("A", 1.0, 1)
    st.addAtoms(["A"] * n, rng.uniform(0, L, (n, 3)), np.zeros(n))
    st.setVelocities(np.arange(n), v0)
    lj = FixLJCut(st, "none")
    lj.setParameter("sig", "A", "A", 1.0)
    lj.setParameter("eps", "A", "A", 0.0)
    st.activateFix(lj)
    nh = FixNoseHoover(st, "nvt", "all")
    nh.setTemperature(T, tau)
    st.activateFix(nh)
    IntegratorVerlet(st).run(steps)
    c = oracle.NoseHooverChain(T, tau, 3 * n, 1.0, dt)
    ke = float(np.sum(v0 ** 2))
    c.prepare(ke)
    scale, most = 1.0, 0.0
    for _ in range(steps):
        for init in (True, False):
            c.ke = ke
            f = c.integrate(init)
            most = max(most, abs(np.log(f)))
            scale *= f
            ke *= f * f
    assert (most > 1.0 / 64) == (tau == 0.01)  # the side of the range that is meant
    v = st.getAtoms()[1]
    # each step rounds the velocities and the scale factor to FP32
    assert np.max(np.abs(v - scale * v0)) < 2 * steps * 2.0 ** -23 * np.abs(v0).max()
