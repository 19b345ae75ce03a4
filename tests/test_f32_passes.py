"""The FP32 passes: the host emulation runs the code of the device library.
Their task sizes are those of the FP32 rule (buffers of 48 KB, which for the
x-forward pass hold the staged rows of two inputs as well, and up to 2048
points), there is one slot record for both precisions, and an evaluation on
grids with odd rows, halves and one-stage axes matches the oracle at the FP32
tolerances of the launch-shape tests."""
import glob
import os

import numpy as np
import pytest

import cases
from oracle import functional as fn
from profess_b200 import native

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "profess_b200", "csrc")


def test_one_slot_record():
    text = [open(p).read() for p in glob.glob(os.path.join(CSRC, "**", "*.cu*"), recursive=True)]
    for name in ("struct SlotDev {", "struct Ctl {", "struct Task {", "struct Args {"):
        assert sum(t.count(name) for t in text) == 1, name


def _slot(eng, n, kinetic):
    cell, _, _, c = cases.golden_case("wgc_al4_fcc" if kinetic == "wgc" else "wt_al4_displaced")
    kin = fn.KEDF_WGC if kinetic == "wgc" else fn.KEDF_WT
    f = cases.functional_for(cell, n, kin, c["alpha"], c["beta"])
    return cell, f, cases.engine_slot(eng, f, cell, precision=native.FP32)


def _check_shape(eng, n, kinetic):
    _, _, s = _slot(eng, n, kinetic)
    try:
        nf, n1 = 8 if kinetic == "wgc" else 4, n[0]  # the x-forward buffers have room for four ion species
        fit = [r for r in range(1, 33) if r * n1 <= 2048]
        want = max(r for r in fit if nf * r * n1 * 8 + 2 * (2 * r * n1 * 4) <= 48 * 1024)
        assert eng.shape(s)["xfwd_row_pairs"] == want
    finally:
        eng.slot_destroy(s)


def _check_eval(eng, n, kinetic):
    cell, f, s = _slot(eng, n, kinetic)
    try:
        rho = cases.random_density(n, cell.num_electrons, cell.vol, seed=3, amp=0.2)
        pot, et = eng.calculate_potential_plus(s, rho)
        po, eo = fn.calculate_potential_plus(f, rho)
        assert np.abs(pot - po).max() < 1e-5 * np.abs(po).max()
        assert np.abs(et - eo).max() < 2e-5
    finally:
        eng.slot_destroy(s)


SHAPES = [((96, 6, 8), "wt"), ((48, 5, 6), "wgc")]
GRIDS = [((12, 9, 15), "wt"), ((5, 9, 10), "wt"), ((48, 5, 6), "wgc"), ((7, 9, 5), "wgc")]


@pytest.mark.parametrize("n,kinetic", SHAPES)
def test_f32_shape_emulated(emu_engine, n, kinetic):
    _check_shape(emu_engine, n, kinetic)


@pytest.mark.parametrize("n,kinetic", GRIDS)
def test_f32_passes_emulated(emu_engine, n, kinetic):
    _check_eval(emu_engine, n, kinetic)


@pytest.mark.gpu
@pytest.mark.parametrize("n,kinetic", SHAPES)
def test_f32_shape(gpu_engine, n, kinetic):
    _check_shape(gpu_engine, n, kinetic)


@pytest.mark.gpu
@pytest.mark.parametrize("n,kinetic", GRIDS)
def test_f32_passes(gpu_engine, n, kinetic):
    _check_eval(gpu_engine, n, kinetic)
