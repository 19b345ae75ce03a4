"""The evaluation at the edges of the FP64 passes' work split, against the
oracle: one-stage x axes (a radix-1 second stage), M = n / R odd and even in
the x-forward pass's last stage, odd n2 and an odd half (a last pair with one
row, pairs across two z), n3 = 4 (halves of two), odd n3 (no row split), and
(y, z) planes that take the split path (WT and WGC).  Tolerances: those of the other evaluation tests."""
import numpy as np
import pytest

import cases
from oracle import functional as fn
from profess_b200 import native

GRIDS = [(5, 6, 8), (12, 9, 10), (27, 14, 6), (35, 15, 18), (42, 10, 4), (16, 12, 15), (36, 21, 14)]
PLANES = [("wt", (4, 135, 240)), ("wgc", (4, 90, 120))]


def _check(eng, n, kinetic):
    cell, _, _, c = cases.golden_case("wgc_al4_fcc" if kinetic == "wgc" else "wt_al4_displaced")
    kin = fn.KEDF_WGC if kinetic == "wgc" else fn.KEDF_WT
    f = cases.functional_for(cell, n, kin, c["alpha"], c["beta"])
    s = eng.slot_create(n, cell.lattice, kinetic=kin, alpha=f.alpha, beta=f.beta, rho0=f.rho_s, rho_s=f.rho_s,
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
def test_grid_edges_emulated(emu_engine, n):
    _check(emu_engine, n, "wt")


@pytest.mark.parametrize("kinetic,n", PLANES)
def test_split_planes_emulated(emu_engine, kinetic, n):
    _check(emu_engine, n, kinetic)


@pytest.mark.gpu
@pytest.mark.parametrize("n", GRIDS)
def test_grid_edges(gpu_engine, n):
    _check(gpu_engine, n, "wt")


@pytest.mark.gpu
@pytest.mark.parametrize("kinetic,n", PLANES)
def test_split_planes(gpu_engine, kinetic, n):
    _check(gpu_engine, n, kinetic)
