"""Molecule form at the sizes where its list build and its pair grid change
shape: the smallest box it takes (2 m + 1 cells a side), one and two rounds of
the pair grid, a ragged last block -- forces against the per-site form."""
import numpy as np
import pytest

from md_engine_b200 import systems

pytestmark = pytest.mark.gpu


def _pairs(x, sysd, cut):
    """oxygen pairs (self pairs with them) within `cut` give or take the edge's
    rounding, and per molecule the sum of 2 C |q q'| / r^3, the most a unit of
    separation changes its Coulomb forces"""
    nmol, near, sure, stiff = len(x) // 4, 0, 0, np.zeros(len(x))
    m = np.arange(len(x)) // 4
    for i in range(0, nmol, 128):
        d = x[4 * i:4 * (i + 128), None] - x[None]
        d -= sysd.L * np.round(d / sysd.L)
        r2 = (d ** 2).sum(2)
        oo = r2[::4, ::4]
        near += int((oo < cut ** 2 + 1e-3).sum())
        sure += int((oo < cut ** 2 - 1e-3).sum())
        rows = slice(4 * i, 4 * i + len(r2))
        r2[m[rows, None] == m[None]] = np.inf
        stiff[rows] = (2 * 332.06 * np.abs(sysd.q[rows, None] * sysd.q[None]) / r2 ** 1.5).sum(1)
    return near, sure, stiff.reshape(-1, 4).sum(1)


@pytest.mark.parametrize("nmol", [730, 1001, 3552, 3601])
def test_molecule_form_matches_per_site_form(nmol):
    sysd = systems.water_tip4p2005(nmol=nmol, seed=nmol)
    f = []
    for form in (1, 2):
        st, _ = systems.build_water_state(sysd, rcut=9.0, skin=1.0, grid=64, alpha=0.3)
        st.pairForm = form
        st.prepare()
        if form == 2:
            near, sure, stiff = _pairs(st.getAtoms()[0], sysd, 9.0 + 1.0 + 2 * (0.9572 + 1e-3))
            # the molecule list holds every pair of oxygens within its radius
            assert sure - nmol <= int(st.molListEntries) <= near - nmol  # FP32 at the edge
        st.computeForces()
        f.append(st.getAtoms()[2])
    rms = np.sqrt(np.mean(np.sum(f[0] ** 2, 1)))
    # the forms round a separation differently, by up to half an ulp of L for
    # each of its two ends: the stiffest contact of a molecule times that,
    # beside the sums' own rounding
    tol = 2e-5 * rms + np.repeat(stiff, 4) * 2.0 ** -23 * sysd.L[0]
    assert np.all(np.linalg.norm(f[1] - f[0], axis=1) < tol)
