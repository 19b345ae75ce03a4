"""The launch shape that the engine reports, pinned again, launches the same
blocks: every kernel of an evaluation keeps its grid, block size and shared
memory."""
import json

import pytest

import cases
from oracle import functional as fn
from profess_b200 import native


def _launches(eng, slot, rho, path):
    import torch
    from torch.profiler import ProfilerActivity, profile
    eng.calculate_potential_plus(slot, rho)
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
        eng.calculate_potential_plus(slot, rho)
        torch.cuda.synchronize()
    p.export_chrome_trace(str(path))
    out = []
    for e in json.load(open(path))["traceEvents"]:
        a = e.get("args", {})
        if e.get("cat") == "kernel" and "ofdft" in e["name"]:
            out.append((e["ts"], e["name"], tuple(a["grid"]), tuple(a["block"]), a.get("shared memory")))
    return [x[1:] for x in sorted(out)]


@pytest.mark.gpu
@pytest.mark.parametrize("n,kinetic,prec", [((64, 64, 64), 4, native.FP64), ((32, 32, 32), 4, native.FP64),
                                            ((45, 45, 45), 4, native.FP64), ((36, 36, 40), 5, native.FP64),
                                            ((96, 96, 96), 4, native.FP64), ((48, 48, 48), 4, native.FP32)])
def test_reported_shape_pinned_again(gpu_engine, tmp_path, n, kinetic, prec):
    import torch
    torch.zeros(1, device="cuda")
    cell, _, _, c = cases.golden_case("wgc_al4_fcc" if kinetic == 5 else "wt_al4_displaced")
    f = cases.functional_for(cell, n, fn.KEDF_WGC if kinetic == 5 else fn.KEDF_WT, c["alpha"], c["beta"])
    s = cases.engine_slot(gpu_engine, f, cell, precision=prec)
    try:
        rho = cases.random_density(n, cell.num_electrons, cell.vol, seed=2)
        before = _launches(gpu_engine, s, rho, tmp_path / "a.json")
        assert any("yzpass" in x[0] for x in before)
        shape = gpu_engine.shape(s)
        gpu_engine.set_shape(s, **shape)
        assert gpu_engine.shape(s) == shape
        assert _launches(gpu_engine, s, rho, tmp_path / "b.json") == before
    finally:
        gpu_engine.slot_destroy(s)
