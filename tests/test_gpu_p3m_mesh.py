"""The library's own FFT of the P3M solve at every mesh side it serves, against
the FP64 restatement: charges alone (no pair fix), so that the forces are the
reciprocal part."""
import numpy as np
import pytest

from md_engine_b200 import Bounds, FixChargeEwald, State, Vector

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", [32, 64, 128])
@pytest.mark.parametrize("n", [2, 777])
def test_p3m_forces_by_mesh(oracle, mesh, n):
    rng = np.random.default_rng(mesh + n)
    L = 20.0
    x = np.asarray(rng.uniform(0.0, L, (n, 3)), np.float32).astype(np.float64)
    q = np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
    q[-1] -= q.sum()
    alpha = 1.0 if mesh == 32 else 1.5
    st = State()
    st.units.setLJ()
    st.bounds = Bounds(st, lo=Vector(0, 0, 0), hi=Vector(L, L, L))
    st.rCut, st.padding, st.dt = 3.0, 0.3, 0.001
    st.atomParams.addSpecies(handle="A", mass=1.0, atomicNum=1)
    st.addAtoms(["A"] * n, x, q)
    ew = FixChargeEwald(st, "charge", "all")
    ew.setParameters(mesh, mesh, mesh, 3.0, 5)
    ew.setAlpha(alpha)
    st.activateFix(ew)
    st.prepare()
    st.computeForces()
    f = st.getAtoms()[2]
    ref = oracle.p3m_forces(x, q, np.zeros(3), np.full(3, L), (mesh,) * 3, alpha, qqr_to_eng=1.0)
    # FP32: a position is off by up to 2^-24 L / 2 in a cell of L / mesh, which
    # shifts a stencil weight (slope below 1 per cell) by up to mesh 2^-25, 4e-6
    # at 128; the mesh sums and transforms add a few 1e-6
    rms = np.sqrt(np.mean(np.sum(ref ** 2, 1)))
    assert np.max(np.linalg.norm(f - ref, axis=1)) < 5e-5 * rms
