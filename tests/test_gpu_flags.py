"""lbm_geometry_flags where other CUDA work has left its marks: an unread error of someone else's call, and a device
pool with no room for the call's scratch."""
import numpy as np
import pytest

from limited_pool import cudart, empty_pool
from pv2013_gb300 import cases

pytestmark = pytest.mark.gpu


def test_flags_with_someone_elses_error_unread(engine):
    geom = cases.vessel(4001).geometry()
    want = geom.flags()
    assert cudart().cudaSetDevice(4096) != 0       # leaves its error for whoever asks
    got = geom.flags()
    left = cudart().cudaGetLastError()
    assert np.array_equal(got, want) and left != 0     # answered, and the error is still its owner's


def test_flags_without_scratch(engine):
    geom = cases.bifurcation().geometry()
    want = geom.flags()
    with empty_pool(1 << 20) as full:
        got = geom.flags() if full else None
    if not full:
        pytest.skip("the pool's size limit is not enforced")
    assert np.array_equal(got, want)
