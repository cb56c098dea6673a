"""Voxelizer on facet normals at the ends of the FP64 range, where products with them under- or overflow: flags equal
to the oracle's every-triangle-for-every-column loop."""
import numpy as np
import pytest

from pv2013_gb300 import Geometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [5e-324, 1e-320, 1e-310, 1e-300, 1e-200, 1e200, 1e300, 1e306, 1.7e308])
def test_extreme_normals_match_oracle(oracle_mod, scale):
    O = oracle_mod
    dims, s, mn = (11, 13, 70), 0.5, (-3.0, 2.0, 10.0)
    rng = np.random.default_rng(7)
    p = rng.uniform(0, 1, (400, 1, 3)) * np.array(dims)
    x = (p + rng.normal(size=(400, 3, 3)) * 3.0) * s + np.array(mn)
    n = np.cross(x[:, 1] - x[:, 0], x[:, 2] - x[:, 0])
    n /= np.linalg.norm(n, axis=1, keepdims=True)
    n[::3, :2] = 0.0                             # horizontal facets: the crossing test's terms are z products alone
    n[::3, 2] = 1.0
    x[::3, 1:, 2] = x[::3, :1, 2]
    t = np.concatenate([x.reshape(400, 9), n * scale], axis=1)
    bb, d = O.explicit_grid((mn, dims), s)
    ref = O.voxelize(t, bb, s, d, binned=False)
    got = Geometry(t, s, grid=(mn, dims)).flags()
    assert np.array_equal(got, ref.reshape(got.shape))
