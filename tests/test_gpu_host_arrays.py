"""Host arrays in and out, below and above the length that is copied in
several threads: what comes back is what went in, rounded to FP32."""
import numpy as np
import pytest

from md_engine_b200 import Bounds, FixLJCut, IntegratorVerlet, State, Vector

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 44000, 90001, 175001])
def test_round_trip(n):
    rng = np.random.default_rng(n)
    L = 80.0
    st = State()
    st.units.setLJ()
    st.bounds = Bounds(st, lo=Vector(0, 0, 0), hi=Vector(L, L, L))
    st.rCut, st.padding, st.dt = 0.5, 0.5, 0.001
    st.atomParams.addSpecies("A", 1.0, 1)
    x0, v0 = rng.uniform(0, L, (n, 3)), rng.standard_normal((n, 3))
    st.addAtoms(["A"] * n, x0, np.zeros(n))
    lj = FixLJCut(st, "none")
    lj.setParameter("sig", "A", "A", 0.1)
    lj.setParameter("eps", "A", "A", 0.0)
    st.activateFix(lj)
    st.prepare()
    x, v = rng.uniform(0, L, (n, 3)), rng.standard_normal((n, 3))
    st.putAtoms(positions=x)
    st.putAtoms(velocities=v)
    xg, vg, fg = st.getAtoms()
    f32 = lambda a: a.astype(np.float32).astype(np.float64)  # noqa: E731
    assert np.array_equal(xg, f32(x)) and np.array_equal(vg, f32(v)) and not fg.any()
    out = IntegratorVerlet(st).runHost(0, x0, v0)
    assert np.array_equal(out["pos"], f32(x0)) and np.array_equal(out["vel"], f32(v0)) and not out["force"].any()
