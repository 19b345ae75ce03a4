"""Rounding error of the FP64 potential against 80-bit values: less than three
quarters of the oracle's (NumPy/SciPy in 64 bits).

Most of it comes from the von Weizsaecker term, whose Laplacian multiplies the
transform's errors by up to the largest |G|^2; they are of the size of what is
transformed.  The engine transforms sqrt(rho) without its mean, which leaves
about a third of its size for these densities (sqrt(rho) varies by a third),
so with transforms of a like error the ratio is near a third, and near one
without the shift."""
import dataclasses

import numpy as np
import pytest
import scipy.fft as sfft

import cases
from oracle import functional as fn

LD = np.longdouble
CASES = [((48, 40, 36), "wt"), ((45, 50, 27), "ab"), ((40, 36, 45), "wgc")]


def _exact(f, rho):
    """calculate_potential_plus in 80 bits (dE/dsqrt(rho)); f's tables are its inputs."""
    third = LD(1) / 3
    c = lambda v: LD(np.float64(v))  # noqa: E731

    def fw(x):
        return sfft.rfftn(x, axes=(1, 2, 0), norm="forward")

    def bw(x):
        return sfft.irfftn(x, s=(f.n[1], f.n[2], f.n[0]), axes=(1, 2, 0), norm="forward")

    r, g2, K = rho.astype(LD), f.qtab.astype(LD) ** 2, f.kernel.astype(LD)
    vh = bw(np.where(g2 > 0, 4 * LD(np.pi) * fw(r) / np.where(g2 > 0, g2, LD(1)), 0))
    r13 = r ** third
    rs = c(0.62035049089940009) / r13
    sr, lr = np.sqrt(rs), np.log(rs)
    vxc = c(-0.98474502184269641) * r13 + np.where(
        rs < 1, lr * (c(3.11e-2) + c(1.33333333333333333e-3) * rs) + c(-5.83666666666666666e-2) + c(-8.4e-3) * rs,
        (c(-1.423e-1) + c(-0.174798948333333333) * sr + c(-6.325709333333333333e-2) * rs)
        / (1 + c(1.0529) * sr + c(3.334e-1) * rs) ** 2)
    a, b = (LD(5) / 6, LD(5) / 6) if f.alpha == f.beta else (LD(f.alpha), LD(f.beta))
    if f.kinetic == fn.KEDF_WT:
        nl = a * r ** (a - 1) * bw(fw(r ** b) * K[0]) + b * r ** (b - 1) * bw(fw(r ** a) * K[0])
    else:
        th, nl = r - LD(f.rho_s), 0
        for x, y in ((a, b), (b, a)):
            F, Ft, t0 = fw(r ** x), fw(th * r ** x), fw(th * th * r ** x / 2)
            w, w2, p3 = bw(K[0] * F + K[1] * Ft + K[2] * t0), bw(K[1] * F + K[3] * Ft), bw(K[2] * F)
            nl = nl + r ** (y - 1) * (y * w + (r + y * th) * w2 + th * (r + y * th / 2) * p3)
    pot = f.ion_pot.astype(LD) + vh + vxc + 5 * third * c(fn.C_TF) * r13 ** 2 + c(fn.C_TF) * nl
    sq = np.sqrt(r)
    return 2 * sq * pot + bw(fw(sq) * g2)


def _check(eng, n, kind):
    kin = fn.KEDF_WGC if kind == "wgc" else fn.KEDF_WT
    cell, _, _, c = cases.golden_case("wgc_al4_fcc" if kind == "wgc" else "wt_al4_displaced")
    alpha, beta = (0.9, 5.0 / 3.0 - 0.9) if kind == "ab" else (c["alpha"], c["beta"])
    f = cases.functional_for(cell, n, kin, alpha, beta)
    # |G| of a cube, whose reciprocal vectors are the same in 64 and 80 bits
    h = np.float64(2.0 * np.pi / 8.0)
    m = [np.arange(n[0] // 2 + 1)] + [np.where(np.arange(k) > k // 2, np.arange(k) - k, np.arange(k)) for k in n[1:]]
    q = np.sqrt((LD(h) * m[0])[:, None, None] ** 2 + (LD(h) * m[1])[None, :, None] ** 2
                + (LD(h) * m[2])[None, None, :] ** 2)
    f80 = dataclasses.replace(f, qtab=q)
    f64 = dataclasses.replace(f, qtab=q.astype(np.float64))
    rho = cases.random_density(n, cell.num_electrons, cell.vol, seed=3, amp=0.25)
    ex = _exact(f80, rho)
    po, _ = fn.calculate_potential_plus(f64, rho)
    s = eng.slot_create(n, 8.0 * np.eye(3), kinetic=kin, alpha=alpha, beta=beta, rho0=f.rho_s, rho_s=f.rho_s)
    try:
        eng.set_kernel(s, f.kernel)
        eng.set_ion_potential(s, f.ion_pot)
        pot, _ = eng.calculate_potential_plus(s, rho)
    finally:
        eng.slot_destroy(s)
    rms = lambda x: float(np.sqrt(((x - ex) ** 2).mean()))  # noqa: E731
    assert rms(pot) < 0.75 * rms(po)


@pytest.mark.parametrize("n,kind", CASES)
def test_potential_accuracy_emulated(emu_engine, n, kind):
    _check(emu_engine, n, kind)


@pytest.mark.gpu
@pytest.mark.parametrize("n,kind", CASES)
def test_potential_accuracy(gpu_engine, n, kind):
    _check(gpu_engine, n, kind)
