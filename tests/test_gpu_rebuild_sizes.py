"""The neighbour list at cell counts around the tiles of the cell scan, and
the pair forces at the sizes where the automatic lanes per atom change."""
import numpy as np
import pytest

from md_engine_b200 import Bounds, FixLJCut, State, Vector
from tests.helpers import neighbor_cut, oracle_nlist_for

pytestmark = pytest.mark.gpu


def _state(n, L, rcut, skin, seed):
    rng = np.random.default_rng(seed)
    k = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = (g[rng.permutation(len(g))[:n]] + 0.5 + rng.uniform(-0.2, 0.2, (n, 3))) * (L / k)
    st = State()
    st.units.setLJ()
    st.bounds = Bounds(st, lo=Vector(0, 0, 0), hi=Vector(L, L, L))
    st.rCut, st.padding, st.dt = rcut, skin, 0.001
    st.atomParams.addSpecies("A", 1.0, 1)
    st.addAtoms(["A"] * n, pos, np.zeros(n))
    lj = FixLJCut(st, "lj")
    lj.setParameter("sig", "A", "A", 1.0)
    lj.setParameter("eps", "A", "A", 1.0)
    st.activateFix(lj)
    st.prepare()
    return st


# cells a side 20 (one tile), 21 (two, the second nearly empty), 32 (exactly four), 33
@pytest.mark.parametrize("side", [20, 21, 32, 33])
def test_list_across_scan_tiles(oracle, side):
    n, rcut, skin = 2 * side ** 3, 1.5, 0.2
    L = side * (1.7 / 2) * 1.0001
    st = _state(n, L, rcut, skin, side)
    assert int(st.cellsPerSide) == side
    x = st.getAtoms()[0].astype(np.float32)
    c, nb, _ = st.getNeighborList()
    co, no = oracle_nlist_for(oracle, x, np.zeros(3), np.full(3, L), neighbor_cut(rcut, skin), ids=np.arange(n))[:2]
    assert np.array_equal(c, co)
    for i in range(0, n, 97):
        assert np.array_equal(np.sort(nb[i, :c[i]]), np.sort(no[i, :co[i]]))


# 126 tiles (a block for each), 130 (two to a block), 256 (two to each of the
# most blocks): a dilute box of few small clumps
@pytest.mark.parametrize("side", [101, 102, 128])
def test_list_of_a_large_dilute_box(oracle, side):
    rng = np.random.default_rng(side)
    rcut, skin, L = 1.5, 0.2, side * 1.7 * 1.0001
    pos = (rng.uniform(0, L, (500, 1, 3)) + rng.uniform(-1.5, 1.5, (500, 6, 3))).reshape(-1, 3) % L
    n = len(pos)
    st = State()
    st.units.setLJ()
    st.bounds = Bounds(st, lo=Vector(0, 0, 0), hi=Vector(L, L, L))
    st.rCut, st.padding, st.dt = rcut, skin, 0.001
    st.atomParams.addSpecies("A", 1.0, 1)
    st.addAtoms(["A"] * n, pos, np.zeros(n))
    lj = FixLJCut(st, "none")
    lj.setParameter("sig", "A", "A", 0.1)
    lj.setParameter("eps", "A", "A", 0.0)
    st.activateFix(lj)
    st.prepare()
    assert int(st.cellsPerSide) == side
    x = st.getAtoms()[0].astype(np.float32)
    c, nb, _ = st.getNeighborList()
    co, no = oracle_nlist_for(oracle, x, np.zeros(3), np.full(3, L), neighbor_cut(rcut, skin), ids=np.arange(n))[:2]
    assert np.array_equal(c, co)
    for i in range(n):
        assert np.array_equal(np.sort(nb[i, :c[i]]), np.sort(no[i, :co[i]]))


@pytest.mark.parametrize("n", [1000, 3000, 7000, 15000, 20000])
def test_forces_at_each_team_size(oracle, n):
    L = (n / 0.8) ** (1 / 3)
    st = _state(n, L, 2.5, 0.3, n)
    st.computeForces()
    x, _, f = st.getAtoms()
    c, nb, _ = st.getNeighborList()
    prm = oracle.lj_params(1, {(0, 0): 1.0}, {(0, 0): 1.0}, 2.5)
    ref = oracle.pair_forces(x, np.zeros(n, int), np.zeros(n), prm, np.full(3, L), c, nb)["f"]
    rms = np.sqrt(np.mean(np.sum(ref ** 2, 1)))
    assert np.max(np.linalg.norm(f - ref, axis=1)) < 2e-4 * rms


# four, three, two warps and one warp per cell on 148 SMs, about five atoms in a cell
@pytest.mark.parametrize("side", [9, 11, 13, 15])
def test_list_with_several_warps_per_cell(oracle, side):
    n, rcut, skin = 5 * side ** 3, 1.5, 0.2
    L = side * (1.7 / 2) * 1.0001
    st = _state(n, L, rcut, skin, side)
    st.gridStencil = 2
    st.prepare()
    assert int(st.cellsPerSide) == side
    x = st.getAtoms()[0].astype(np.float32)
    c, nb, _ = st.getNeighborList()
    co, no = oracle_nlist_for(oracle, x, np.zeros(3), np.full(3, L), neighbor_cut(rcut, skin), ids=np.arange(n))[:2]
    assert np.array_equal(c, co)
    for i in range(0, n, 97):
        assert np.array_equal(np.sort(nb[i, :c[i]]), np.sort(no[i, :co[i]]))
