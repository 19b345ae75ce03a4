"""Accuracy of the FP64 epilogue's powers of the density (the device's functions),
against 80-bit values.

On a uniform density every transform is exact (sums of equal numbers on a grid
of a power of two), so the potential is that of one point: with a constant
kernel K it is vxc + 5/3 C_TF rho^(2/3) + C_TF K (alpha + beta) rho^(alpha + beta - 1).

* Over the whole range of the fast inverse cube root and beyond its ends
  (rho from 1e-70 to 1e70), no potential is further off than 16 half units in
  the last place of the sum of its terms' sizes: at most 16 roundings (and
  powers of at most 2 units) lie on the way of any term.
* In the unequal-exponent functional K is made large, so that the powers and
  1/rho = (rho^(-1/3))^3 decide the error.  With every operation an independent
  rounding (RMS 0.64e-16 of its result), rho^(-1/3) 0.5e-16, the two powers 0.7e-16
  each in halves of the sum, 1/rho is off by 1.75e-16 and the potential by 2.4e-16;
  the bound leaves a quarter: 3.0e-16.  (With rho^(-1/3) as a square of
  rho^(-1/6), 1/rho is off by 3.5e-16 and the potential by 3.9e-16.)
"""
import numpy as np
import pytest

from oracle.consts import C_TF
from profess_b200 import native

LD = np.longdouble
N = (4, 4, 4)


def _slot(eng, alpha, beta, k):
    s = eng.slot_create(N, 8.0 * np.eye(3), alpha=alpha, beta=beta, rho0=0.03, rho_s=0.03, mu=0.0)
    eng.set_kernel(s, np.full((3, 4, 4), k))
    eng.set_ion_potential(s, np.zeros(N))
    return s


def _terms(rho, a, b, k):
    c = lambda v: LD(np.float64(v))  # noqa: E731
    rho, third = LD(rho), LD(1) / 3
    r13 = rho ** third
    rs = c(0.62035049089940009) / r13
    x = c(-0.98474502184269641) * r13
    if rs < 1:
        lr = np.log(rs)
        t = [x, lr * c(3.11e-2), lr * c(1.33333333333333333e-3) * rs, c(-5.83666666666666666e-2), c(-8.4e-3) * rs]
    else:
        sr = np.sqrt(rs)
        den = (1 + c(1.0529) * sr + c(3.334e-1) * rs) ** 2
        t = [x, c(-1.423e-1) / den, c(-0.174798948333333333) * sr / den, c(-6.325709333333333333e-2) * rs / den]
    t += [5 * third * c(C_TF) * r13 ** 2, c(C_TF) * c(k) * (a + b) * rho ** (a + b - 1)]
    return t


def _errors(eng, alpha, beta, k, densities, exact):
    s = _slot(eng, alpha, beta, k)
    out = []
    try:
        for rho in densities:
            pot, _ = eng.calculate_potential_plus(s, np.full(N, rho), opt_sqrt=False)
            t = _terms(rho, *exact, k)
            out.append(float((LD(pot[1, 2, 3]) - sum(t)) / sum(abs(x) for x in t)))
    finally:
        eng.slot_destroy(s)
    return np.abs(np.array(out))


@pytest.mark.gpu
def test_powers(gpu_engine):
    rng = np.random.default_rng(1)
    wide = 10.0 ** np.concatenate([np.arange(-70, 71, 2.5), rng.uniform(-62, 62, 100)])
    e = _errors(gpu_engine, 5.0 / 6.0, 5.0 / 6.0, 0.25, wide, (LD(5) / 6, LD(5) / 6))
    assert e.max() < 16 * 1.11e-16
    usual = 10.0 ** rng.uniform(-5, 1, 400)
    e = _errors(gpu_engine, 0.9, 0.7, 64.0, usual, (LD(np.float64(0.9)), LD(np.float64(0.7))))
    assert np.sqrt((e ** 2).mean()) < 3.0e-16
