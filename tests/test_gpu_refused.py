"""A step whose launch is refused (its stream holds an invalidated capture) fails and leaves the handle's state: the
steps after it give the bits of an undisturbed run."""
import ctypes as C

import numpy as np
import pytest

from pv2013_gb300 import Simulation, _capi, cases

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
def test_refused_launch_leaves_the_state(cudart, precision, pattern):
    rt = cudart
    c, geom = small()
    st = new_stream(rt)
    make = lambda s: Simulation(geom, c.tau, c.boundary_specs(geom), precision=precision, pattern=pattern,  # noqa: E731
                                stream=s)
    sim, ref = make(st.value), make(None)
    sim.step(3)
    assert rt.cudaStreamSynchronize(st) == 0
    assert rt.cudaStreamBeginCapture(st, 1) == 0
    assert rt.cudaStreamSynchronize(st) != 0     # not allowed on a capturing stream: the capture is invalid now
    rt.cudaGetLastError()
    with pytest.raises(_capi.LbmError):
        sim.step(1)
    graph = C.c_void_p()
    assert rt.cudaStreamEndCapture(st, C.byref(graph)) != 0
    rt.cudaGetLastError()
    assert sim.info().steps_done == 3
    sim.step(4)
    ref.step(7)
    assert np.array_equal(sim.fields()[0], ref.fields()[0])
    sim.close()
    rt.cudaStreamDestroy(st)
