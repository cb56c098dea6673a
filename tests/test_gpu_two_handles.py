"""Distinct handles are independent whatever their block sizes: FP64 simulations of one and of four warps per block,
which share a kernel, stepped in turn and from two threads, give the bits of separate runs."""
import threading

import numpy as np
import pytest
import torch

from pv2013_gb300 import Simulation, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Q", [19, 27])
@pytest.mark.parametrize("pattern", ["pull", "aa"])
def test_block_sizes_in_turn_and_from_threads(Q, pattern):
    c = cases.pipe(radius=7.0, length=33.0, ny=41, nxz=19)
    geom = c.geometry()
    specs = c.boundary_specs(geom) if Q == 19 else ()
    steps = 8000

    def make(warps, stream=None):
        return Simulation(geom, c.tau, specs, Q=Q, precision="f64", pattern=pattern, warps_per_block=warps,
                          stream=stream.cuda_stream if stream else None)

    ref = make(4)
    ref.step(steps)
    want = ref.fields()[0]
    small, large = make(1), make(4)
    for _ in range(100):
        small.step(1)
        large.step(1)
    streams = [torch.cuda.Stream() for _ in range(3)]
    sims = [make(w, s) for w, s in zip((1, 4, 8), streams)]
    errors = []

    def work(sim, n):
        try:
            for _ in range(n // 40):
                sim.step(40)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(s, steps)) for s in sims]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for s in sims:
        assert np.array_equal(s.fields()[0], want)
    small.step(steps - 100)
    large.step(steps - 100)
    assert np.array_equal(small.fields()[0], want) and np.array_equal(large.fields()[0], want)
