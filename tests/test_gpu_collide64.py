"""FP64 collision on any populations: the AA even launch (node-local) against
the reference's expressions evaluated operation by operation in numpy
(Simulation.cpp:21-179), bit for bit -- flow-like values, and values outside
the range of the shared reciprocal: zero, subnormal, huge, infinite, NaN."""
import numpy as np
import pytest

from pv2013_gb300 import LatticeModel, Simulation, cases

pytestmark = pytest.mark.gpu
HEADER = 88          # LBMCKPT2: the plane-major populations follow


def collide_ref(f, Q, om):
    m = LatticeModel(Q)
    c, w = m.c, m.w
    s = lambda idx: sum((f[i] for i in idx[1:]), f[idx[0]])  # noqa: E731  left to right
    rho = s(list(range(Q)))
    if Q == 19:
        groups = [([0, 6, 7, 8, 9], [1, 10, 11, 12, 13]), ([2, 6, 10, 14, 15], [3, 7, 11, 16, 17]),
                  ([4, 8, 12, 14, 16], [5, 9, 13, 15, 17])]
    else:
        groups = [([1, 7, 8, 11, 13, 19, 21, 23, 25], [2, 9, 10, 12, 14, 20, 22, 24, 26]),
                  ([3, 7, 9, 15, 16, 19, 21, 24, 26], [4, 8, 10, 17, 18, 20, 22, 23, 25]),
                  ([5, 11, 12, 15, 17, 19, 22, 23, 26], [6, 13, 14, 16, 18, 20, 21, 24, 25])]
    ux, uy, uz = [(s(p) - s(n)) / rho for p, n in groups]
    usq = ux * ux + uy * uy + uz * uz
    out = np.empty_like(f)
    for q in range(Q):
        du = ux * float(c[q][0]) + uy * float(c[q][1]) + uz * float(c[q][2])
        feq = w[q] * rho * (1.0 + 3.0 * du + 4.5 * du * du - 1.5 * usq)
        out[q] = om * feq + (1.0 - om) * f[q]
    return out


@pytest.mark.parametrize("Q", [19, 27])
@pytest.mark.parametrize("staging", [0, 1])
def test_collision_any_populations_bit_exact(tmp_path, Q, staging):
    c = cases.pipe(radius=7.0, length=33.0, ny=41, nxz=19)
    sim = Simulation(c.geometry(), 0.83, (), Q=Q, precision="f64", pattern="aa", staging=staging,
                     corrections=3)     # boundary nodes collide what their slots hold, like every other node
    path = str(tmp_path / "a.ckpt")
    sim.checkpoint(path)
    raw = np.fromfile(path, dtype=np.uint8)
    f = raw[HEADER:].view(np.float64).reshape(Q, -1)
    n = f.shape[1]
    rng = np.random.default_rng(Q + staging)
    f[:] = LatticeModel(Q).w[:, None] * (1.0 + 0.2 * rng.standard_normal((Q, n)))
    special = [0.0, -0.0, 5e-324, 1e-310, -1e-300, 1e-250, 1e200, -1e160, 1e308, np.inf, -np.inf, np.nan, 1.0, 2.0 ** -101]
    for k, v in enumerate(special):
        f[rng.integers(Q), k::40] = v            # one population of many nodes
        f[:, 20 + k::61] = v                     # every population of others
    f[:, 3::50] *= 1e-290
    with np.errstate(over="ignore"):
        f[:, 4::50] *= 1e120
    f[1:, 5::50] = 0.0                           # one population alone: j = rho
    old = f.copy()
    raw.tofile(path)
    sim.restart(path)
    sim.step(1)
    sim.checkpoint(path)
    new = np.fromfile(path, dtype=np.uint8)[HEADER:].view(np.float64).reshape(Q, -1)
    with np.errstate(all="ignore"):
        ref = collide_ref(old, Q, 1.0 / 0.83)
    ref = ref[LatticeModel(Q).opp]               # the launch writes f*_q to slot opp(q)
    same = ((new == ref) | (np.isnan(new) & np.isnan(ref))).all(axis=0)
    kept = ((new == old) | (np.isnan(new) & np.isnan(old))).all(axis=0)
    assert (same | kept).all()                   # every node is collided, or no fluid node
    assert same.sum() >= sim.info().n_nodes
    assert np.isfinite(ref).all(axis=0).sum() > n // 4
