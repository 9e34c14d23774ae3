"""Host arrays in and out, below and above the length that is copied in
several threads and the length that crosses in one piece: what comes back is
what went in, rounded to FP32."""
import threading

import numpy as np
import pytest

from md_engine_b200 import Bounds, FixLJCut, IntegratorVerlet, State, Vector

pytestmark = pytest.mark.gpu


def _f32(a):
    return a.astype(np.float32).astype(np.float64)


def _state(n, seed, L=80.0):
    rng = np.random.default_rng(seed)
    st = State()
    st.units.setLJ()
    st.bounds = Bounds(st, lo=Vector(0, 0, 0), hi=Vector(L, L, L))
    st.rCut, st.padding, st.dt = 0.5, 0.5, 0.001
    st.atomParams.addSpecies("A", 1.0, 1)
    x0, v0 = rng.uniform(0, L, (n, 3)), rng.standard_normal((n, 3))
    st.addAtoms(["A"] * n, x0, np.zeros(n))
    st.setVelocities(np.arange(n), v0)
    lj = FixLJCut(st, "none")
    lj.setParameter("sig", "A", "A", 0.1)
    lj.setParameter("eps", "A", "A", 0.0)
    st.activateFix(lj)
    st.prepare()
    return st, x0, v0


# 21,845 atoms cross to the host in one piece, more in pieces of 10,922; an array
# of 32,768 atoms to the device; in a host-buffer run the three results of
# 233,016 atoms at once, else arrays of 349,525 atoms in one piece
@pytest.mark.parametrize("n", [1, 255, 21845, 21846, 32769, 44000, 90001, 175001, 233016, 233017, 350001])
def test_round_trip(n):
    rng, L = np.random.default_rng(n + 1), 80.0
    st, x0, v0 = _state(n, n)
    x, v = rng.uniform(0, L, (n, 3)), rng.standard_normal((n, 3))
    st.putAtoms(positions=x)
    st.putAtoms(velocities=v)
    xg, vg, fg = st.getAtoms()
    assert np.array_equal(xg, _f32(x)) and np.array_equal(vg, _f32(v)) and not fg.any()
    st.putAtoms(positions=x0, velocities=v0)
    xg, vg, fg = st.getAtoms()
    assert np.array_equal(xg, _f32(x0)) and np.array_equal(vg, _f32(v0)) and not fg.any()
    out = IntegratorVerlet(st).runHost(0, x, v)
    assert np.array_equal(out["pos"], _f32(x)) and np.array_equal(out["vel"], _f32(v)) and not out["force"].any()


def test_states_share_their_staging():
    """a state's first getAtoms takes no device memory once another state of
    the process has crossed arrays of that length"""
    torch = pytest.importorskip("torch")
    states = [_state(60000, k)[0] for k in range(4)]
    states[0].getAtoms()
    free = torch.cuda.mem_get_info()[0]
    for st in states[1:]:
        st.getAtoms()
    assert torch.cuda.mem_get_info()[0] == free


def test_states_of_several_threads():
    """more threads than slots of the shared staging, each with its own state"""
    states = [_state(20000 + 501 * k, k) for k in range(7)]
    bad = []

    def work(k):
        st, _, v0 = states[k]
        rng = np.random.default_rng(100 + k)
        for _ in range(10):
            x = rng.uniform(0, 80.0, v0.shape)
            st.putAtoms(positions=x)
            xg, vg, _ = st.getAtoms()
            if not (np.array_equal(xg, _f32(x)) and np.array_equal(vg, _f32(v0))):
                bad.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(states))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
