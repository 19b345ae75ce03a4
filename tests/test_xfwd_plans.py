"""The x-forward pass's own plans (last stage of radix 4 at most, or 1) and its
two ways of taking the functional's powers, against the oracle: axes of one
stage (6, 14), whose last radix would be 5 or 7 (25, 49: a stage of radix 1),
of three stages where two would do (64); equal and unequal WT exponents and WGC;
the row split and whole planes (odd n3); a density of 1e-80 at some points,
outside the range of the fast inverse cube root.  Tolerances: those of the
other evaluation tests."""
import numpy as np
import pytest

import cases
from oracle import functional as fn

GRIDS = [(6, 9, 10), (14, 9, 15), (25, 6, 8), (49, 5, 6), (64, 6, 5)]
KINDS = ["wt", "ab", "wgc"]


def _check(eng, n, kind, tiny):
    cell, _, _, c = cases.golden_case("wgc_al4_fcc" if kind == "wgc" else "wt_al4_displaced")
    kin = fn.KEDF_WGC if kind == "wgc" else fn.KEDF_WT
    alpha, beta = (1.2, 5.0 / 3.0 - 1.2) if kind == "ab" else (c["alpha"], c["beta"])
    f = cases.functional_for(cell, n, kin, alpha, beta)
    s = eng.slot_create(n, cell.lattice, kinetic=kin, alpha=alpha, beta=beta, rho0=f.rho_s, rho_s=f.rho_s,
                        ion_ion=f.ion_ion)
    try:
        eng.set_kernel(s, f.kernel)
        eng.set_ion_potential(s, f.ion_pot)
        rho = cases.random_density(n, cell.num_electrons, cell.vol, seed=3, amp=0.2)
        if tiny:
            rho[1::3, ::2, 1::4] = 1e-80
        pot, et = eng.calculate_potential_plus(s, rho)
        po, eo = fn.calculate_potential_plus(f, rho)
        assert np.abs(pot - po).max() < 1e-11 * np.abs(po).max()
        assert np.abs(et - eo).max() < 1e-10 * max(1.0, np.abs(eo).max())
    finally:
        eng.slot_destroy(s)


CASES = [(n, k, False) for n in GRIDS for k in KINDS] + [((12, 9, 10), "wt", True), ((12, 9, 15), "wt", True)]


@pytest.mark.parametrize("n,kind,tiny", CASES)
def test_xfwd_plans_emulated(emu_engine, n, kind, tiny):
    _check(emu_engine, n, kind, tiny)


@pytest.mark.gpu
@pytest.mark.parametrize("n,kind,tiny", CASES)
def test_xfwd_plans(gpu_engine, n, kind, tiny):
    _check(gpu_engine, n, kind, tiny)
