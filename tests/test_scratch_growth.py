"""The first forces and stress of an engine allocate no device memory beyond
what the set-up took: the transfer scratch grows in steps, and the Ewald sum's
share of it is the same with and without forces."""
import pytest

from profess_b200 import cell as pcell
from profess_b200 import native
from profess_b200 import workloads as wl


@pytest.mark.gpu
def test_first_forces_allocate_nothing():
    import torch
    from torch.profiler import ProfilerActivity, profile
    torch.zeros(1, device="cuda")
    c = wl.fcc_al((2, 2, 2), sigma_ang=0.05, grid=(32, 32, 32), seed=3)

    def calls(fn):
        with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
            fn()
            torch.cuda.synchronize()
        return {e.name for e in p.events()}

    eng = native.Engine()
    try:
        s = pcell.setup_slot(eng, c)
        eng.set_input(s, wl.initial_density(c, seed=1))
        eng.start_solve(s, None, native.ntn_options(conv_check=native.CONV_POT, pot_tol=1e-3))
        while eng.run(8):
            pass
        first = calls(lambda: (eng.forces(s, c.nion), eng.stress(s)))
        assert any("cudaLaunchKernel" in n for n in first)  # the calls are recorded
        assert not any(n.startswith(("cudaMalloc", "cudaFree")) for n in first)
        other = native.Engine()  # a set-up is recorded to allocate
        try:
            assert any(n.startswith("cudaMalloc") for n in calls(lambda: pcell.setup_slot(other, c)))
        finally:
            other.close()
    finally:
        eng.close()
