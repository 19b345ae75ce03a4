"""The device Ewald sum (energy, forces, stress) against the oracle at the
edges of its work split: one ion (a partner only in its own images), a
skewed cell (image ranges that differ by axis), ions given outside [0, 1),
a row longer than the 128 m3 values kept between ion chunks, and more ions
than one chunk of 256.

Tolerances: those of the other Ewald tests (1e-10 of max(1, |E|) Ha, 1e-10
Ha/bohr); the stress within 1e-12 Ha/bohr^3, 1e-10 of its size (about 1e-2).
"""
import numpy as np
import pytest

from oracle import ewald as oew
from oracle import stress as ost
from profess_b200 import cell as pcell
from profess_b200 import workloads as wl


def _cell(name):
    if name == "one ion":
        c = wl.fcc_al((1, 1, 1), grid=(10, 10, 10))
        c.frac, c.species_of_ion = c.frac[:1] + 0.3, c.species_of_ion[:1]
        return c
    if name == "skewed":
        c = wl.fcc_al((1, 2, 1), sigma_ang=0.1, grid=(8, 12, 10), seed=4)
        c.lattice = (np.eye(3) + np.array([[0.0, 0.45, 0.2], [0.0, 0.0, -0.35], [0.1, 0.0, 0.0]])) @ c.lattice
        c.frac = c.frac + np.array([1.0, -2.0, 0.0])
        return c
    if name == "long":
        return wl.fcc_al((1, 1, 24), sigma_ang=0.05, grid=(8, 8, 128), seed=2)
    return wl.fcc_al((5, 4, 4), sigma_ang=0.05, grid=(24, 20, 20), seed=3)  # 320 ions


NAMES = ["one ion", "skewed", "long", "two chunks"]


def _check(eng, name):
    c = _cell(name)
    s = pcell.setup_slot(eng, c)
    try:
        e, f = eng.ewald(s, c.nion)
        eo, fo = oew.ewald(c.lattice, c.frac, c.charges(), True)
        assert abs(e - eo) < 1e-10 * max(1.0, abs(eo))
        assert np.abs(f - fo).max() < 1e-10
        e2, none = eng.ewald(s, c.nion, want_forces=False)
        assert none is None and e2 == e
        if c.nion <= 100:
            rho = np.full(c.grid, c.num_electrons / c.vol)
            _, parts = eng.stress(s, rho=rho, terms=True)
            assert np.abs(parts["Ewald"] - ost.ewald_stress(c.lattice, c.frac, c.charges())).max() < 1e-12
    finally:
        eng.slot_destroy(s)


@pytest.mark.parametrize("name", NAMES)
def test_ewald_edges_emulated(emu_engine, name):
    _check(emu_engine, name)


@pytest.mark.gpu
@pytest.mark.parametrize("name", NAMES)
def test_ewald_edges(gpu_engine, name):
    _check(gpu_engine, name)


def _check_stress_rows(eng, reps, grid):
    """The stress reduction's rows: two species, more z positions than threads
    of a block, more ions than one chunk; every term against the oracle's
    tensor (1e-10 Ha/bohr^3, as the other stress tests)."""
    import cases
    from oracle import cellsetup as cs, functional as fn, kedf_kernels as kk
    c = wl.fcc_al(reps, sigma_ang=0.1, grid=grid, seed=7)
    c.species = [wl.al_species(), wl.mg_species()]
    c.species_of_ion = np.arange(c.nion) % 3 % 2
    osp = [cs.species_from_table(*wl.heine_abarenkov_table(z, rc, 0.1), n)
           for z, rc, n in ((3.0, 1.15, "Al"), (2.0, 1.3, "Mg"))]
    oc = cs.Cell(lattice=c.lattice, frac=c.frac, species_of_ion=c.species_of_ion, species=osp)
    rho_avg = oc.num_electrons / oc.vol
    kern = kk.wt_kernel(cs.q_table(oc.recip, *grid), rho_avg, c.alpha, c.beta, 1.0, 1.0)[None]
    f = fn.Functional(kinetic=4, n=grid, dv=oc.vol / np.prod(grid), qtab=cs.q_table(oc.recip, *grid), kernel=kern,
                      ion_pot=cs.ion_potential_real(oc, *grid), ion_ion=0.0, lam=1.0, mu=1.0, alpha=c.alpha,
                      beta=c.beta, rho_s=rho_avg)
    s = pcell.setup_slot(eng, c)
    try:
        rho = cases.random_density(grid, oc.num_electrons, oc.vol, seed=4, amp=0.2)
        got = eng.stress(s, rho=rho)
        assert np.abs(got - ost.stress(oc, f, rho)).max() < 1e-10
    finally:
        eng.slot_destroy(s)


def test_stress_rows_emulated(emu_engine):
    _check_stress_rows(emu_engine, (1, 1, 2), (10, 9, 21))


@pytest.mark.gpu
@pytest.mark.parametrize("reps,grid", [((1, 1, 2), (10, 9, 21)), ((1, 1, 8), (16, 15, 135)),
                                       ((4, 4, 5), (20, 18, 27))])
def test_stress_rows(gpu_engine, reps, grid):
    _check_stress_rows(gpu_engine, reps, grid)
