"""The device STL reader without device memory: a file that the host grammar parses anyway (it holds a NUL byte) is
read all the same, any other is refused with LBM_ERR_NOMEM."""
import numpy as np
import pytest

from limited_pool import empty_pool
from pv2013_gb300 import Reader, _capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("facets", [3, 9000])
def test_files_without_device_memory(tmp_path, engine, facets):
    tris = np.random.default_rng(facets).normal(size=(facets, 12))
    plain, nul = tmp_path / "a.stl", tmp_path / "b.stl"
    Reader.writeSTLASCII(plain, tris)
    text = bytearray(plain.read_bytes())
    text[len(text) * 3 // 4] = 0
    nul.write_bytes(text)
    with empty_pool(256) as full:
        if full:
            with pytest.raises(_capi.LbmError) as e:
                Reader.readSTLASCIIDevice(plain)
            got, on_device = Reader.readSTLASCIIDevice(nul)
    if not full:
        pytest.skip("the pool's size limit is not enforced")
    assert "LBM_ERR_NOMEM" in str(e.value)
    assert not on_device and np.array_equal(got, Reader.readSTLASCII(nul), equal_nan=True)


def test_a_directory_is_refused(tmp_path, engine):
    with pytest.raises(_capi.LbmError):
        Reader.readSTLASCIIDevice(tmp_path)
