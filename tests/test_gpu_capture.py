"""lbm_sim_step on a stream that the caller captures: the captured launches have plain edges and replay to the bits of
direct steps."""
import ctypes as C

import numpy as np
import pytest

from pv2013_gb300 import Simulation, cases

pytestmark = pytest.mark.gpu


@pytest.fixture
def cudart(engine):
    rt = C.CDLL("libcudart.so.13")              # the runtime the library is linked with
    return rt


def new_stream(rt):
    s = C.c_void_p()
    assert rt.cudaStreamCreateWithFlags(C.byref(s), 1) == 0
    return s


def small():
    c = cases.pipe(radius=7.0, length=33.0, ny=41, nxz=19)
    return c, c.geometry()


@pytest.mark.parametrize("precision,pattern", [("f16s", "aa"), ("f32", "pull"), ("f64", "pull"), ("f64", "aa")])
def test_captured_steps(cudart, precision, pattern):
    rt = cudart
    c, geom = small()
    st = new_stream(rt)
    make = lambda s: Simulation(geom, c.tau, c.boundary_specs(geom), precision=precision, pattern=pattern,  # noqa: E731
                                stream=s)
    sim, ref = make(st.value), make(None)
    sim.step(2)
    graph, ex, n = C.c_void_p(), C.c_void_p(), C.c_size_t()
    assert rt.cudaStreamBeginCapture(st, 1) == 0
    sim.step(3)
    assert rt.cudaStreamEndCapture(st, C.byref(graph)) == 0
    frm, to, edges = (C.c_void_p * 8)(), (C.c_void_p * 8)(), (C.c_ubyte * 64)()
    n.value = 8
    assert rt.cudaGraphGetEdges(graph, frm, to, edges, C.byref(n)) == 0
    assert n.value == 2 and not any(edges)       # full completion, no programmatic dependency
    rt.cudaGraphInstantiate.argtypes = [C.c_void_p, C.c_void_p, C.c_ulonglong]
    assert rt.cudaGraphInstantiate(C.byref(ex), graph, 0) == 0
    assert rt.cudaGraphLaunch(ex, st) == 0
    assert rt.cudaStreamSynchronize(st) == 0
    ref.step(5)
    assert sim.info().steps_done == 5
    assert np.array_equal(sim.fields()[0], ref.fields()[0])
    sim.step(4)                                  # direct (chained) launches again
    ref.step(4)
    assert np.array_equal(sim.fields()[0], ref.fields()[0])
    rt.cudaGraphExecDestroy(ex)
    rt.cudaGraphDestroy(graph)
    sim.close()
    rt.cudaStreamDestroy(st)
