"""The autotuner times what it chooses for, graph replay: every paired candidate is the kernel that graphs replay, none
the chained variant of direct launches."""
import pytest
import torch

from pv2013_gb300 import Simulation, cases

pytestmark = pytest.mark.gpu


def kernels(fn):
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        fn()
        torch.cuda.synchronize()
    return [e.name for e in prof.events() if "k_step2" in e.name]


@pytest.mark.parametrize("precision", ["f16s", "f32"])
def test_candidates_run_unchained(precision):
    torch.zeros(1, device="cuda")
    c = cases.pipe(radius=7.0, length=33.0, ny=41, nxz=19)
    geom = c.geometry()
    sim = Simulation(geom, c.tau, c.boundary_specs(geom), precision=precision, pattern="aa")
    kernels(lambda: sim.step(1))                 # the profiler's first session may record nothing
    direct = kernels(lambda: sim.step(3))
    if not direct:
        pytest.skip("no kernel records from the profiler here")
    assert all("true>" in k or "1>" in k for k in direct), direct[:2]       # direct launches of a small lattice: chained
    timed = kernels(lambda: sim.autotune(launches=2))
    assert len(timed) > 20 and all("false>" in k or "0>" in k for k in timed), timed[:3]
