"""Performance cases of the density-solve engine, through its public entry points.

What a user of the engine has it do, over the sizes of this repository's own
workloads (``profess_b200/workloads.py``: fcc Al cells of 4-500 atoms on
32^3-120^3 grids, hcp Mg up to 1152 atoms on 160x160x256) and odd sizes
between them:

* ``solve``   - density solves to the reference's default tolerance, alone
                (the drop-in ``ProjNormRhoMinimization`` call) or as a batch
                of cells that share every launch;
* ``eval``    - one drop-in ``CalculatePotentialPlus`` call on host arrays;
* ``forces``  - ion forces of a solved density;
* ``stress``  - stress tensor of a solved density;
* ``ions``    - the tables rebuilt after the ions moved (ion potential,
                Ewald energy and forces), read back by a host code.

FP32 slots serve the first phase of mixed-precision solves, so the single
passes are FP64.  Arrays that an FP32 slot computed are returned as FP32.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from profess_b200 import cell as pcell
from profess_b200 import native
from profess_b200 import workloads as wl

C_TF = 2.87123400018819
WGC_TOL, WT_TOL, FP32_TOL = 1.0e-5, 1.0e-5, 3.0e-5


# ----------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest call a host code makes: one 4-atom cell, launch and latency bound
        dict(name="solve 1x al4 32 fp64", kind="solve", metal="al", reps="1x1x1", grid="32x32x32", cells=1,
             prec="fp64", kinetic="wt", mixed=False),
        # a batch of small cells (training-set generation): 16 of them share the launches
        dict(name="solve 16x al4 32 fp64", kind="solve", metal="al", reps="1x1x1", grid="32x32x32", cells=16,
             prec="fp64", kinetic="wt", mixed=False),
        # the headline workload's two precisions: the FP32 phase of a mixed solve, and the plain FP64 solve
        dict(name="solve 16x al256 96 fp32", kind="solve", metal="al", reps="4x4x4", grid="96x96x96", cells=16,
             prec="fp32", kinetic="wt", mixed=False),
        dict(name="solve 16x al256 96 fp64", kind="solve", metal="al", reps="4x4x4", grid="96x96x96", cells=16,
             prec="fp64", kinetic="wt", mixed=False),
        # cells of 32-500 atoms (48^3-120^3) served together
        dict(name="solve 12x al32-500 fp64", kind="solve", metal="al", reps="2x2x2", grid="48x48x48", cells=12,
             prec="fp64", kinetic="wt", mixed=True),
        # hexagonal cells on odd grids with the second-order WGC functional
        dict(name="solve 4x mg72 wgc fp32", kind="solve", metal="mg", reps="3x4x3", grid="63x81x100", cells=4,
             prec="fp32", kinetic="wgc", mixed=False),
        # the largest cell: 1152 atoms, WGC
        dict(name="solve 1x mg1152 wgc fp64", kind="solve", metal="mg", reps="8x8x9", grid="160x160x256", cells=1,
             prec="fp64", kinetic="wgc", mixed=False),
        # drop-in evaluations of a host code: a usual grid, and an odd one with unequal WT exponents
        dict(name="eval al256 96 fp64", kind="eval", metal="al", reps="4x4x4", grid="96x96x96", cells=1,
             prec="fp64", kinetic="wt", mixed=False),
        dict(name="eval 45x50x54 ab fp64", kind="eval", metal="al", reps="2x2x2", grid="45x50x54", cells=1,
             prec="fp64", kinetic="wt_ab", mixed=False),
        # after a solve: the forces of a relaxation or MD step, the stress of a cell relaxation or NPT step
        dict(name="forces al256 96 fp64", kind="forces", metal="al", reps="4x4x4", grid="96x96x96", cells=1,
             prec="fp64", kinetic="wt", mixed=False),
        dict(name="stress al108 72 fp64", kind="stress", metal="al", reps="3x3x3", grid="72x72x72", cells=1,
             prec="fp64", kinetic="wt", mixed=False),
        # the ions moved: every table that depends on them rebuilt
        dict(name="ions al500 120 fp64", kind="ions", metal="al", reps="5x5x5", grid="120x120x120", cells=1,
             prec="fp64", kinetic="wt", mixed=False),
    ]


def _near(rng, n):
    """A 7-smooth grid length near n, often odd."""
    return wl.smooth_size(max(16, n + rng.randint(-4, 6)))


def draw(rng):
    kind = rng.choice(["solve"] * 6 + ["eval"] * 2 + ["forces", "stress", "ions"])
    prec = rng.choice(["fp64", "fp64", "fp32"]) if kind == "solve" else "fp64"
    kinetic = rng.choice(["wt", "wt", "wgc"]) if kind != "eval" else rng.choice(["wt", "wt_ab"])
    points = 10 ** rng.uniform(4.4, 6.6)
    if kinetic == "wgc":
        points = min(points, 2.5e6)
    edge = points ** (1.0 / 3.0)
    per = rng.uniform(20.0, 27.0)  # grid points per conventional cell edge (about 5-6.7 per Angstrom)
    if kinetic == "wgc":
        metal = "mg"
        per_a = per * 3.21 / 4.05
        reps = [max(1, round(edge / per_a + rng.choice([-1, 0, 0, 1]))) for _ in range(2)]
        reps.append(max(1, round(edge / (per_a * 1.624) + rng.choice([-1, 0, 0, 1]))))
        grid = [_near(rng, round(per_a * r * s)) for r, s in zip(reps, (1.0, 1.0, 1.624))]
    else:
        metal = "al"
        reps = [max(1, round(edge / per + rng.choice([-1, 0, 0, 1]))) for _ in range(3)]
        grid = [_near(rng, round(per * r)) for r in reps]
    n = grid[0] * grid[1] * grid[2]
    cells = 1
    if kind == "solve":  # batches as large as the headline one
        room = 14.0e6 / (n * (2.5 if kinetic == "wgc" else 1.0))
        cells = max(1, min(16, int(math.exp(rng.uniform(0.0, math.log(max(1.0, room)))))))
    return dict(kind=kind, metal=metal, reps="x".join(map(str, reps)), grid="x".join(map(str, grid)), cells=cells,
                prec=prec, kinetic=kinetic, mixed=False)


# ----------------------------------------------------------------- inputs
def _ints(text):
    return tuple(int(x) for x in text.split("x"))


def _cells(case, seed):
    out = []
    for k in range(case["cells"]):
        s = 1000 * seed + k
        reps, grid = _ints(case["reps"]), _ints(case["grid"])
        if case["mixed"]:  # 2x2x2 to 5x5x5 conventional cells, lattice within 2 %
            r = 2 + k % 4
            strain = float(np.random.default_rng(s).uniform(-0.02, 0.02))
            out.append(wl.fcc_al((r, r, r), sigma_ang=0.05, strain=strain, seed=s))
        elif case["metal"] == "al":
            out.append(wl.fcc_al(reps, sigma_ang=0.02 if reps == (1, 1, 1) else 0.05, grid=grid, seed=s))
        else:
            out.append(wl.hcp_mg(reps, sigma_ang=0.05, grid=grid, seed=s))
    return out


def _prec(case):
    return native.FP32 if case["prec"] == "fp32" else native.FP64


def _eval_input(case, seed):
    """A host code's arrays for one evaluation: lattice, keKernel, ion potential, density, Ewald energy."""
    rng = np.random.default_rng(seed)
    c = _cells(dict(case, cells=1), seed)[0]
    n1, n2, n3 = c.grid
    alpha, beta = (0.9, 5.0 / 3.0 - 0.9) if case["kinetic"] == "wt_ab" else (5.0 / 6.0, 5.0 / 6.0)
    rho0 = c.num_electrons / c.vol
    ax = [np.arange(n) * (2.0 * math.pi / n) for n in c.grid]

    def waves(count):
        w = np.zeros(c.grid)
        for _ in range(count):
            k = rng.integers(1, 4, size=3)
            ph = rng.uniform(0, 2 * math.pi, size=3)
            w += (np.cos(k[0] * ax[0] + ph[0])[:, None, None] * np.cos(k[1] * ax[1] + ph[1])[None, :, None]
                  * np.cos(k[2] * ax[2] + ph[2])[None, None, :])
        return w / count

    rho = rho0 * (1.0 + 0.6 * waves(4)) * (1.0 + 0.01 * rng.random(c.grid))
    rho *= c.num_electrons / (rho.sum() * c.vol / rho.size)
    vion = 0.4 * waves(4) - 0.1
    q = np.sqrt(_g2(c.lattice, c.grid))
    eta = q / (2.0 * (3.0 * math.pi ** 2 * rho0) ** (1.0 / 3.0))
    with np.errstate(divide="ignore", invalid="ignore"):
        lind = 1.0 / (0.5 + 0.25 * (1.0 - eta ** 2) * np.log((1.0 + eta) / np.abs(1.0 - eta)) / eta)
    lind = np.where(eta < 1e-8, 1.0, np.where(np.abs(eta - 1.0) < 1e-8, 2.0, lind))
    kern = (lind - 3.0 * eta ** 2 - 1.0) * 5.0 / (9.0 * alpha * beta * rho0 ** (alpha + beta - 5.0 / 3.0))
    return dict(grid=c.grid, lattice=c.lattice, vol=c.vol, alpha=alpha, beta=beta, rho0=rho0,
                rho=np.asfortranarray(rho), vion=np.asfortranarray(vion), kern=np.asfortranarray(kern),
                ion_ion=-2.7 * c.nion)


def _g2(lattice, grid):
    """|G|^2 on the half spectrum (n1/2+1, n2, n3)."""
    b = 2.0 * math.pi * np.linalg.inv(lattice).T
    f = [np.arange(n) for n in grid]
    f = [np.arange(grid[0] // 2 + 1)] + [np.where(x > n // 2, x - n, x) for x, n in zip(f[1:], grid[1:])]
    g2 = np.zeros((grid[0] // 2 + 1, grid[1], grid[2]))
    for r in range(3):
        g = b[r, 0] * f[0][:, None, None] + b[r, 1] * f[1][None, :, None] + b[r, 2] * f[2][None, None, :]
        g2 += g * g
    return g2


def prepare(case, seed):
    eng = native.Engine()
    prec = _prec(case)
    st = dict(case=case, eng=eng, f32=prec == native.FP32)
    if case["kind"] == "eval":
        d = _eval_input(case, seed)
        s = eng.slot_create(d["grid"], d["lattice"], alpha=d["alpha"], beta=d["beta"], rho0=d["rho0"],
                            ion_ion=d["ion_ion"], precision=prec)
        eng.set_kernel(s, d["kern"])
        eng.set_ion_potential(s, d["vion"])
        st.update(slot=s, rho=d["rho"])
        return st
    cells = _cells(case, seed)
    slots = [pcell.setup_slot(eng, c, precision=prec) for c in cells]
    tol = FP32_TOL if prec == native.FP32 else WGC_TOL if case["kinetic"] == "wgc" else WT_TOL
    st.update(cells=cells, slots=slots,
              opts=native.ntn_options(conv_check=native.CONV_POT, pot_tol=tol, stall_line=6))
    if case["kind"] == "ions":
        # the next geometry: the same cell, its ions displaced otherwise
        st["moved"] = _cells(case, seed + 500009)[0].frac
        return st
    if case["kind"] == "solve" and case["cells"] == 1:
        st["rho"] = wl.initial_density(cells[0], seed=seed)
        return st
    for k, (s, c) in enumerate(zip(slots, cells)):
        eng.set_input(s, wl.initial_density(c, seed=1000 * seed + k))
    if case["kind"] != "solve":  # forces and stress are of a solved density
        _solve_batch(st)
    return st


# ----------------------------------------------------------------- one pass
def _solve_batch(st):
    eng = st["eng"]
    for s in st["slots"]:
        eng.start_solve(s, None, st["opts"])
    while eng.run(8):
        pass


def _own(st, a):
    return a.astype(np.float32) if st["f32"] else a


def run(st):
    eng, kind = st["eng"], st["case"]["kind"]
    if kind == "eval":
        pot, et = eng.calculate_potential_plus(st["slot"], st["rho"])
        return {"potential": _own(st, pot), "energy": _own(st, et)}
    if kind == "forces":
        return {"forces": _own(st, eng.forces(st["slots"][0], st["cells"][0].nion))}
    if kind == "stress":
        return {"stress": _own(st, eng.stress(st["slots"][0]))}
    if kind == "ions":
        c, s = st["cells"][0], st["slots"][0]
        eng.build_ion_potential(s, st["moved"], c.species_of_ion, c.species)
        e, f = eng.ewald(s, c.nion)
        return {"ewald": np.array([e]), "ewald_forces": f, "potential": _own(st, eng.download(s, 2))}
    if st["case"]["cells"] == 1:  # the drop-in call: host density in and out
        rho, e, _ = eng.proj_norm_rho_minimization(st["slots"][0], st["rho"], st["opts"])
        return {"rho0": _own(st, rho), "energy0": _own(st, e)}
    _solve_batch(st)
    out = {}
    for k, s in enumerate(st["slots"]):
        rho, e, _ = eng.result(s)
        out["rho%d" % k] = _own(st, rho)
        out["energy%d" % k] = _own(st, e)
    return out


# ----------------------------------------------------------------- minimal work
def work(case):
    """One evaluation reads the density (and, in a solve, the search direction), the ion potential and the
    kernel planes and writes the potential; its 3D transforms are nf forward and nf inverse.  A solve to
    these tolerances takes about 85 evaluations (WT), 120 (WGC), 70 in FP32."""
    b = 4 if case["prec"] == "fp32" else 8
    grids = [wl.smooth_size(24 * (2 + k % 4)) for k in range(case["cells"])]
    pts = (sum(g ** 3 for g in grids) if case["mixed"] else case["cells"] * math.prod(_ints(case["grid"])))
    nf, planes = {"wt": (3, 1), "wt_ab": (4, 1), "wgc": (8, 4)}[case["kinetic"]]
    lg = math.log2(pts / case["cells"])
    fft = 2.5 * lg * pts
    one_b, one_f = b * pts * (4 + planes / 2.0), 2 * nf * fft + 80 * pts
    kind = case["kind"]
    if kind == "solve":
        evals = 70 if b == 4 else 120 if case["kinetic"] == "wgc" else 85
        return {"bytes": evals * one_b, "flops": evals * one_f}
    if kind == "eval":
        return {"bytes": one_b + 8 * pts, "flops": one_f}
    nion = math.prod(_ints(case["reps"])) * (4 if case["metal"] == "al" else 2)
    sten = 1000.0 * nion
    if kind == "forces":
        return {"bytes": b * pts + 8 * 3 * nion, "flops": 2 * fft + 8 * sten}
    if kind == "stress":
        return {"bytes": b * pts, "flops": one_f + nf * fft + 40 * pts}
    return {"bytes": 2 * 8 * pts, "flops": 2 * fft + 2 * sten}


# ----------------------------------------------------------------- 64-bit values
def exact(case, seed):
    if case["kind"] == "eval":
        return _exact_eval(_eval_input(case, seed))
    if case["kind"] == "ions":
        c = _cells(case, seed + 500009)[0]
        e, f = _exact_ewald(c.lattice, c.frac, c.charges())
        return {"ewald": np.array([e]), "ewald_forces": f, "potential": None}
    return None  # an iterative solve, or sums over one


def _exact_eval(d):
    """Potential dE/dsqrt(rho) and the energy table of CalculatePotentialPlus with the WT functional."""
    grid, rho = d["grid"], np.ascontiguousarray(d["rho"].T)  # (z, y, x): the last axis is halved
    g2 = np.ascontiguousarray(_g2(d["lattice"], grid).T)
    kern, vion = d["kern"].T, d["vion"].T

    def conv(x, k):
        return np.fft.irfftn(np.fft.rfftn(x) * k, s=rho.shape, axes=(0, 1, 2))

    a, b = d["alpha"], d["beta"]
    sq, r13 = np.sqrt(rho), np.cbrt(rho)
    with np.errstate(divide="ignore"):
        vh = conv(rho, np.where(g2 > 0, 4 * math.pi / np.where(g2 > 0, g2, 1.0), 0.0))
    lap = conv(sq, g2)
    pb = conv(rho ** b, kern)
    pa = conv(rho ** a, kern)
    rs = 0.62035049089940009 / r13
    ln, s = np.log(rs), np.sqrt(rs)
    den = 1.0 + 1.0529 * s + 0.3334 * rs
    ec = np.where(rs < 1, ln * (3.11e-2 + 2e-3 * rs) - 4.8e-2 - 1.16e-2 * rs, -0.1423 / den)
    vc = np.where(rs < 1, ln * (3.11e-2 + 1.33333333333333333e-3 * rs) - 5.83666666666666666e-2 - 8.4e-3 * rs,
                  (-0.1423 - 0.174798948333333333 * s - 6.325709333333333333e-2 * rs) / den ** 2)
    vnl = C_TF * (a * rho ** (a - 1) * pb + b * rho ** (b - 1) * pa)
    pot = vion + vh - 0.98474502184269641 * r13 + vc + 5.0 / 3.0 * C_TF * r13 ** 2 + vnl
    e = np.array([0, 0, (rho * vion).sum(), 0.5 * (rho * vh).sum(), (rho * (ec - 0.73855876638202234 * r13)).sum(),
                  0, C_TF * (rho * r13 ** 2).sum(), 0.5 * (sq * lap).sum(), C_TF * (rho ** a * pb).sum()])
    e[1] = e[6:].sum()
    e *= d["vol"] / rho.size
    e[5] = d["ion_ion"]
    e[0] = e[1:6].sum()
    return {"potential": (2.0 * sq * pot + lap).T, "energy": e}


def _exact_ewald(lattice, frac, z):
    """Ewald energy and forces of point charges in a neutralising background."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t = lambda x: torch.tensor(np.asarray(x), dtype=torch.float64, device=dev)  # noqa: E731
    n, vol, inv = len(z), abs(np.linalg.det(lattice)), np.linalg.inv(lattice)
    eta = math.sqrt(math.pi) * (n / vol ** 2) ** (1.0 / 6.0)
    rcut, gcut = 7.0 / eta, 14.0 * eta

    def shell(heights, cut):
        r = [np.arange(-m, m + 1) for m in (int(math.ceil(cut / h)) + 1 for h in heights)]
        return np.stack([x.ravel() for x in np.meshgrid(*r, indexing="ij")], axis=1).astype(float)

    pos, q = t(frac @ lattice.T), t(z)
    img = t(shell(1.0 / np.sqrt((inv ** 2).sum(axis=1)), rcut) @ lattice.T)
    f, e = torch.zeros(n, 3, dtype=torch.float64, device=dev), 0.0
    for i in range(n):
        d = pos[None] + img[:, None] - pos[i]
        r = d.norm(dim=-1)
        ok = (r > 1e-12) & (r < rcut)
        d, r, w = d[ok], r[ok], q.expand(len(img), n)[ok] * q[i]
        ec = torch.erfc(eta * r) / r
        e += 0.5 * float((w * ec).sum())
        g = -w * (ec + 2.0 * eta / math.sqrt(math.pi) * torch.exp(-(eta * r) ** 2)) / r ** 2
        f[i] = (g[:, None] * d).sum(0)
    g = shell(np.sqrt((lattice ** 2).sum(axis=0)) ** -1 * 2 * math.pi, gcut) @ (2 * math.pi * inv)
    g2 = (g ** 2).sum(axis=1)
    keep = (g2 > 0) & (g2 <= gcut ** 2)
    g, g2 = t(g[keep]), t(g2[keep])
    w = torch.exp(-g2 / (4 * eta * eta)) / g2
    ph = g @ pos.T
    c, s = torch.cos(ph), torch.sin(ph)
    sr, si = c @ q, s @ q
    e += 2 * math.pi / vol * float((w * (sr ** 2 + si ** 2)).sum())
    e += -eta / math.sqrt(math.pi) * float((q * q).sum()) - 0.5 * math.pi / eta ** 2 / vol * float(q.sum()) ** 2
    f += 4 * math.pi / vol * q[:, None] * ((w * sr)[:, None] * s - (w * si)[:, None] * c).T @ g
    return e, f.cpu().numpy()
