"""A last pair of rows that has only one row: the half plane (FP64, even n3) or
the whole plane (odd n3) has an odd number of rows.  The fields of the missing
row are zero whatever the functional makes of a zero density: with a negative
Wang-Teter exponent, 0^beta is infinite, and must not reach the row that is
there.  Tolerances: those of the other evaluation tests."""
import numpy as np
import pytest

import cases
from oracle import functional as fn

GRIDS = [(12, 9, 10), (12, 9, 15), (12, 15, 18)]
EXPONENTS = [(2.0, -1.0 / 3.0), (0.9, 5.0 / 3.0 - 0.9), (5.0 / 6.0, 5.0 / 6.0)]


def _check(eng, n, alpha, beta):
    cell, _, _, _ = cases.golden_case("wt_al4_displaced")
    f = cases.functional_for(cell, n, fn.KEDF_WT, alpha, beta)
    s = eng.slot_create(n, cell.lattice, kinetic=fn.KEDF_WT, alpha=alpha, beta=beta, rho0=f.rho_s, rho_s=f.rho_s,
                        ion_ion=f.ion_ion)
    try:
        eng.set_kernel(s, f.kernel)
        eng.set_ion_potential(s, f.ion_pot)
        rho = cases.random_density(n, cell.num_electrons, cell.vol, seed=3, amp=0.2)
        pot, et = eng.calculate_potential_plus(s, rho)
        po, eo = fn.calculate_potential_plus(f, rho)
        assert np.abs(pot - po).max() < 1e-11 * np.abs(po).max()
        assert np.abs(et - eo).max() < 1e-10 * max(1.0, np.abs(eo).max())
    finally:
        eng.slot_destroy(s)


@pytest.mark.parametrize("n", GRIDS)
@pytest.mark.parametrize("alpha,beta", EXPONENTS)
def test_missing_row_emulated(emu_engine, n, alpha, beta):
    _check(emu_engine, n, alpha, beta)


@pytest.mark.gpu
@pytest.mark.parametrize("n", GRIDS)
@pytest.mark.parametrize("alpha,beta", EXPONENTS)
def test_missing_row(gpu_engine, n, alpha, beta):
    _check(gpu_engine, n, alpha, beta)
