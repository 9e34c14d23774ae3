"""The kernel that joins one step's second half to the next one's first, at
one, two and the most blocks of its cluster and just past them: one chunk of
five steps (four turns) against five chunks of one step (none)."""
import numpy as np
import pytest

from md_engine_b200 import Bounds, FixLJCut, FixNoseHoover, IntegratorVerlet, State, Vector

pytestmark = pytest.mark.gpu

STEPS = 5


@pytest.mark.parametrize("nh", [True, False])
@pytest.mark.parametrize("n", [1, 512, 513, 8192, 8193])
def test_ideal_gas_steps_joined_or_not(n, nh):
    rng = np.random.default_rng(n)
    x0 = rng.uniform(1.0, 39.0, (n, 3)).astype(np.float32).astype(np.float64)
    v0 = rng.standard_normal((n, 3)).astype(np.float32).astype(np.float64)
    out = []
    for interval in (STEPS, 1):
        st = State()
        st.units.setLJ()
        st.bounds = Bounds(st, lo=Vector(0, 0, 0), hi=Vector(40, 40, 40))
        st.rCut, st.padding, st.dt, st.periodicInterval = 1.0, 0.5, 0.005, interval
        st.atomParams.addSpecies("A", 1.0, 1)
        st.addAtoms(["A"] * n, x0, np.zeros(n))
        st.setVelocities(np.arange(n), v0)
        lj = FixLJCut(st, "none")
        lj.setParameter("sig", "A", "A", 1.0)
        lj.setParameter("eps", "A", "A", 0.0)
        st.activateFix(lj)
        if nh:
            fix = FixNoseHoover(st, "nvt", "all")
            fix.setTemperature(0.7, 0.5)
            st.activateFix(fix)
        IntegratorVerlet(st).run(STEPS)
        out.append(st.getAtoms()[:2])
    # without forces only the scale factor can differ, by its rounding to FP32
    # where the kinetic sum's order moved it across a rounding boundary
    assert np.max(np.abs(out[0][1] - out[1][1])) <= (STEPS * 2.0 ** -23 * np.abs(out[1][1]).max() if nh else 0.0)
    assert np.max(np.abs(out[0][0] - out[1][0])) <= (STEPS * 2.0 ** -18 if nh else 0.0)
