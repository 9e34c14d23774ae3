"""The kernel that joins one step's second half to the next one's first, at
one, two and the most blocks of its cluster and just past them: one chunk of
five steps (four turns) against five chunks of one step (none), without forces
and with them."""
import numpy as np
import pytest

from md_engine_b200 import Bounds, FixChargeEwald, FixLJCut, FixNoseHoover, IntegratorVerlet, State, Vector

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


def _fluid(n, salt, nh, interval):
    """n - 2 (or, n odd, n - 1) atoms on a jittered lattice, alternately charged
    in a salt, the others massless and without forces; a skin that no atom
    leaves in five steps, so that both runs sum the same pairs"""
    rng = np.random.default_rng(n)
    heavy = n - 1 if n % 2 else n - 2
    k = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    L = 1.05 * k
    x = ((g + 0.5 + rng.uniform(-0.06, 0.06, (n, 3))) * 1.05).astype(np.float32).astype(np.float64)
    v = rng.standard_normal((n, 3)).astype(np.float32).astype(np.float64)
    st = State()
    st.units.setLJ()
    st.bounds = Bounds(st, lo=Vector(0, 0, 0), hi=Vector(L, L, L))
    st.rCut, st.padding, st.dt, st.periodicInterval = 2.5, 0.6, 0.002, interval
    st.atomParams.addSpecies("A", 1.0, 1)
    st.atomParams.addSpecies("M", 0.0, 1)
    q = np.where(np.arange(n) < heavy, (-1.0) ** g.sum(1), 0.0) if salt else np.zeros(n)
    q[0] -= q.sum()
    st.addAtoms(["A"] * heavy + ["M"] * (n - heavy), x, q)
    st.setVelocities(np.arange(n), v)
    lj = FixLJCut(st, "lj")
    for a, b, eps in (("A", "A", 1.0), ("M", "M", 0.0), ("A", "M", 0.0)):
        lj.setParameter("sig", a, b, 1.0)
        lj.setParameter("eps", a, b, eps)
    st.activateFix(lj)
    if salt:
        ew = FixChargeEwald(st, "charge", "all")
        ew.setParameters(32, 32, 32, 2.5, 5)
        ew.setAlpha(1.0)
        st.activateFix(ew)
    if nh:
        fix = FixNoseHoover(st, "nvt", "all")
        fix.setTemperature(0.7, 0.5)
        st.activateFix(fix)
    return st, heavy


@pytest.mark.parametrize("salt", [False, True])
@pytest.mark.parametrize("nh", [True, False])
@pytest.mark.parametrize("n", [513, 8192])
def test_fluid_steps_joined_or_not(n, nh, salt):
    out = []
    for interval in (STEPS, 1):
        st, heavy = _fluid(n, salt, nh, interval)
        IntegratorVerlet(st).run(STEPS)
        assert st.status()[2] == 1  # one list for the whole run
        out.append(st.getAtoms())
    (xa, va, fa), (xb, vb, fb) = out
    assert not va[heavy:].any() and not vb[heavy:].any()
    rms = np.sqrt(np.mean(np.sum(fb[:heavy] ** 2, 1)))
    # a half kick dropped or doubled would show in what follows
    assert 0.5 * 0.002 * rms > 100 * 1e-5 * np.abs(vb).max()
    if not (nh or salt):
        assert np.array_equal(xa, xb) and np.array_equal(va, vb) and np.array_equal(fa, fb)
        return
    # with a thermostat the scale factor may differ by an ulp, with P3M the
    # charges' spread adds in another order (1e-6 of the forces): a position is
    # off by an ulp at most, which moves a force by the stiffness of its
    # contacts, a few thousand, times 2e-6
    assert np.max(np.abs(va - vb)) < 1e-5 * np.abs(vb).max()
    assert np.max(np.abs(xa - xb)) < 1e-5
    assert np.max(np.linalg.norm(fa - fb, axis=1)) < 1e-3 * rms
