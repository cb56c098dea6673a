"""Paired steps launched one by one (chained launches on lattices of one wave of
blocks) against graph replay, with snapshots and monitors between them: the same
bits, below and above the one-wave size."""
import numpy as np
import pytest

from pv2013_gb300 import Simulation, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pattern", ["aa", "pull"])
@pytest.mark.parametrize("precision,Q", [("f16s", 19), ("bf16s", 19), ("f32", 27)])
@pytest.mark.parametrize("case", ["small", "wave", "large"])
def test_chained_launches_equal_graph_replay(pattern, precision, Q, case):
    c = {"small": lambda: cases.pipe(radius=7.0, length=33.0, ny=41, nxz=19), "wave": lambda: cases.vessel(4005),
         "large": lambda: cases.pipe(radius=40.0, length=300.0, ny=308, nxz=88)}[case]()
    geom = c.geometry()
    specs = c.boundary_specs(geom) if Q == 19 else ()
    a, b, d = [Simulation(geom, c.tau, specs, Q=Q, precision=precision, pattern=pattern) for _ in range(3)]
    for n in (1, 7, 16):
        a.step(n)                                   # launch by launch
        b.step(n, graph=True)
        for _ in range(n):                          # and with a snapshot after every step
            d.step(1)
            d.monitors()
        fa, ra, ua = a.fields()
        assert np.array_equal(fa, b.fields()[0]) and np.array_equal(fa, d.fields()[0])
    assert np.isfinite(fa).all() and a.monitors() == b.monitors()
