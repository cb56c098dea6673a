"""Voxelizer where its cheap bounds meet the exact tests: random triangles on
lattice lines and planes, needles, slivers, point-like projections, crossings
at the test's tolerance, coordinates far from the grid, spacings below the face
nudge -- flags equal to the oracle's every-triangle-for-every-column loop."""
import numpy as np
import pytest

from pv2013_gb300 import Geometry

pytestmark = pytest.mark.gpu


def soup(rng, kind, n, dims, s, mn):
    hi = np.array(dims) * 1.0
    t = np.empty((n, 12))
    p = rng.uniform(-1.5, 1.0, (n, 1, 3)) * 0.2 * hi + rng.uniform(0, 1, (n, 1, 3)) * hi
    v = p + rng.normal(size=(n, 3, 3)) * rng.choice([0.3, 1.0, 4.0, 30.0], (n, 1, 1))
    if kind == "lattice":                        # vertices on lattice points, half of them exactly
        r = rng.random((n, 3, 1)) < 0.6
        v = np.where(r, np.rint(v), v)
    elif kind == "needle":                       # collinear in xy up to a tiny offset, some along an axis
        d = rng.normal(size=(n, 3))
        d[::3, 0] = 0.0
        d[1::3, 1] = 0.0
        a = np.where(rng.random((n, 1)) < 0.5, np.rint(p[:, 0]), p[:, 0])
        off = rng.choice([0.0, 1e-13, 1e-11, 1e-9, 1e-7, 1e-4], (n, 1)) * rng.normal(size=(n, 3))
        v = np.stack([a, a + d * rng.uniform(0.1, 9, (n, 1)), a + d * rng.uniform(0.1, 9, (n, 1)) + off], 1)
    elif kind == "point":                        # vertical line in z
        v[:, 1:, :2] = v[:, :1, :2] + rng.choice([0.0, 1e-12, 1e-8], (n, 1, 1)) * rng.normal(size=(n, 2, 2))
        v[:, :, :2] = np.where(rng.random((n, 1, 1)) < 0.5, np.rint(v[:, :1, :2]), v[:, :, :2])
    elif kind == "tolerance":                    # horizontal facets at a point's height +- the tolerance
        L = (dims[2] - 1) * s
        z = np.rint(v[:, :1, 2:]) + rng.choice([0.0, 1e-7, -1e-7, 1 + 1e-7, 1.0], (n, 1, 1)) * (L + 0.1) / s * \
            (1 + rng.choice([0, 1e-15, -1e-15, 1e-12, -1e-9, 1e-6], (n, 1, 1)))
        v[:, :, 2:] = z
    elif kind == "outside":                      # needles and slivers that start far outside and point at the grid
        d = hi * rng.uniform(0.1, 0.9, (n, 3)) - p[:, 0] * 0
        a = d + rng.choice([-1, 1], (n, 1)) * rng.uniform(30, 5000, (n, 1)) * rng.normal(size=(n, 3)) * [1, 1, 0.01]
        far = a + (a - d) * rng.uniform(0.001, 0.2, (n, 1))
        off = rng.choice([0.0, 1e-11, 1e-8, 1e-5, 0.3], (n, 1)) * rng.normal(size=(n, 3))
        d = np.where(rng.random((n, 1)) < 0.5, np.rint(d), d)
        v = np.stack([a, far, np.where(rng.random((n, 1)) < 0.5, d, a + 0.5 * (far - a)) + off], 1)
    elif kind == "far":
        v = p + rng.normal(size=(n, 3, 3)) * rng.choice([1e3, 3e6, 1e9], (n, 1, 1))
    x = v * s + np.array(mn)
    t[:, :9] = x.reshape(n, 9)
    nrm = np.cross(x[:, 1] - x[:, 0], x[:, 2] - x[:, 0])
    ln = np.linalg.norm(nrm, axis=1, keepdims=True)
    t[:, 9:] = np.where(ln > 0, nrm / np.where(ln > 0, ln, 1), 0.0)
    odd = rng.random(n)
    t[odd < 0.10, 9:] = rng.normal(size=(int((odd < 0.10).sum()), 3))          # a normal of its own
    t[(odd > 0.10) & (odd < 0.15), 11] = 0.0
    t[(odd > 0.15) & (odd < 0.20), 11] *= 1e-14
    return t


@pytest.mark.parametrize("kind", ["any", "lattice", "needle", "point", "tolerance", "far", "outside"])
@pytest.mark.parametrize("dims,s,mn", [((13, 11, 17), 1.0, (0.0, 0.0, 0.0)), ((9, 14, 70), 0.37, (-175.3, 12.7, 1e4)),
                                       ((12, 7, 33), 0.003, (2.0, -1.0, 0.5)), ((1, 2, 3), 0.25, (0.125, 0.0, -4.0))])
def test_triangle_soup_matches_oracle(oracle_mod, kind, dims, s, mn):
    O = oracle_mod
    seed = 1000 * ["any", "lattice", "needle", "point", "tolerance", "far", "outside"].index(kind) + dims[0]
    t = soup(np.random.default_rng(seed), kind, 900, dims, s, mn)
    bb, d = O.explicit_grid((mn, dims), s)
    got = Geometry(t, s, grid=(mn, dims)).flags()
    ref = O.voxelize(t, bb, s, d, binned=False)
    assert np.array_equal(got, ref.reshape(got.shape))
    assert kind in ("needle", "point", "outside") or dims[0] == 1 or 0 < ref.sum() < ref.size
