"""Task and block sizes that a launch takes by what it holds change no bit: a
cell solved alone and the same cell among others of its kind, of another size
and of another functional end on the same density and energies (FP64; the row
split and whole planes, WT with equal and unequal exponents, WGC)."""
import numpy as np
import pytest

from profess_b200 import cell as pcell
from profess_b200 import native
from profess_b200 import workloads as wl

KINDS = [("wt", (30, 42, 70)), ("wt", (27, 25, 45)), ("ab", (20, 36, 24)), ("wgc", (24, 20, 35)), ("wgc", (16, 18, 20))]


def _cell(kind, grid, seed):
    if kind == "wgc":
        return wl.hcp_mg((1, 1, 1), sigma_ang=0.02, grid=grid, seed=seed)
    c = wl.fcc_al((1, 1, 1), sigma_ang=0.02, grid=grid, seed=seed)
    if kind == "ab":
        c.alpha, c.beta = 0.9, 5.0 / 3.0 - 0.9
    return c


@pytest.mark.gpu
@pytest.mark.parametrize("kind,grid", KINDS)
def test_alone_and_among_others(gpu_engine, kind, grid):
    eng = gpu_engine
    opts = native.ntn_options(conv_check=native.CONV_POT, pot_tol=1e-12, max_iter=3)
    others = [(kind, grid)] * 9 + [k for k in KINDS if k != (kind, grid)]
    slots = []
    try:
        for q, (k, g) in enumerate([(kind, grid)] + others):
            c = _cell(k, g, seed=q)
            s = pcell.setup_slot(eng, c)
            slots.append(s)
            eng.set_input(s, wl.initial_density(c, seed=q))

        def solve(which):
            for s in which:
                eng.start_solve(s, None, opts)
            while eng.run(8):
                pass
            rho, e, st = eng.result(slots[0])
            return rho.copy(), e.copy(), st["num_evals"]

        alone, among = solve(slots[:1]), solve(slots)
        assert alone[2] == among[2]
        assert np.array_equal(alone[0], among[0]) and np.array_equal(alone[1], among[1])
    finally:
        for s in slots:
            eng.slot_destroy(s)
