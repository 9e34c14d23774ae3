"""A state prepared a second time after what its neighbour list was sized for
changed -- the lanes per atom, when the charge fix is taken off, and the number
of atoms -- against a state prepared once."""
import numpy as np
import pytest

from md_engine_b200 import Bounds, FixChargeEwald, FixLJCut, State, Vector

pytestmark = pytest.mark.gpu

RCUT, SKIN = 2.8, 0.3


def _side(n):
    return (n / 0.75) ** (1 / 3)


def _positions(n, seed):
    rng = np.random.default_rng(seed)
    k = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)
    return (g[rng.permutation(len(g))[:n]] + 0.5 + rng.uniform(-0.2, 0.2, (n, 3))) * (_side(n) / k)


def _state(pos, side, n_charged):
    """neutral Lennard-Jones sites A, then n_charged charged sites B without one"""
    n, L = len(pos), side
    st = State()
    st.units.setLJ()
    st.bounds = Bounds(st, lo=Vector(0, 0, 0), hi=Vector(L, L, L))
    st.rCut, st.padding, st.dt = RCUT, SKIN, 0.001
    for h in "AB":
        st.atomParams.addSpecies(h, 1.0, 1)
    q = np.zeros(n)
    q[n - n_charged:] = np.where(np.arange(n_charged) % 2 == 0, 1.0, -1.0)
    st.addAtoms(["A"] * (n - n_charged) + ["B"] * n_charged, pos, q)
    lj = FixLJCut(st, "lj")
    for h, eps in (("A", 1.0), ("B", 0.0)):
        lj.setParameter("sig", h, h, 0.8)
        lj.setParameter("eps", h, h, eps)
    st.activateFix(lj)
    return st


def _compare(st, ref):
    assert int(st.nThreadPerAtom) == int(ref.nThreadPerAtom)
    assert int(st.nlistCapacity) % int(st.nThreadPerAtom) == 0
    out = []
    for s in (st, ref):
        s.computeForces()
        c, nb, _ = s.getNeighborList()
        out.append((c, [np.sort(nb[i, :c[i]]) for i in range(len(c))], s.getAtoms()[2]))
        assert s.status()[0] == 0
    assert np.array_equal(out[0][0], out[1][0])
    assert all(np.array_equal(a, b) for a, b in zip(out[0][1], out[1][1]))
    # the same pairs in the same rows: only the order of a row's sums may differ
    rms = np.sqrt(np.mean(np.sum(out[1][2] ** 2, 1)))
    assert np.max(np.abs(out[0][2] - out[1][2])) < 1e-5 * rms


# lanes per atom 8 with the charge fix and 16 without it, 4 and 8; seeds whose
# first list has a row capacity that is no multiple of the second's lanes
@pytest.mark.parametrize("n,seed,teams", [(6000, 10, (8, 16)), (12000, 3, (4, 8))])
def test_charge_fix_taken_off(n, seed, teams):
    pos = _positions(n, seed)
    st = _state(pos, _side(n), n // 2)
    ew = FixChargeEwald(st, "charge", "all")
    ew.setParameters(32, 32, 32, RCUT, 5)
    ew.setAlpha(1.0)
    st.activateFix(ew)
    st.prepare()
    assert int(st.nThreadPerAtom) == teams[0] and int(st.nlistCapacity) % teams[1] != 0
    st.deactivateFix(ew)
    st.prepare()
    ref = _state(pos, _side(n), n // 2)
    ref.prepare()
    assert int(ref.nThreadPerAtom) == teams[1]
    _compare(st, ref)


def test_atoms_added():
    pos = _positions(5000, 3)
    st = _state(pos[:1500], _side(5000), 0)
    st.prepare()
    st.addAtoms(["A"] * 3500, pos[1500:], np.zeros(3500))
    st.prepare()
    ref = _state(pos, _side(5000), 0)
    ref.prepare()
    _compare(st, ref)
