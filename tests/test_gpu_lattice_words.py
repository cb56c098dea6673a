"""Lattice construction at the edges of its 32-bit words: axes of 29 to 66 points,
runs that start, end or fill a word, fluid on every face of the grid, on both run
axes.  Random populations are written through a checkpoint: streaming and
bounce-back of every node against the same on the dense grid in numpy, and the
paired piece tables of every size against one node per lane."""
import numpy as np
import pytest

from pv2013_gb300 import Geometry, LatticeModel, Simulation, synth_cylinder

pytestmark = pytest.mark.gpu


def box(lo, hi):
    c = np.array([[x, y, z] for x in (lo[0], hi[0]) for y in (lo[1], hi[1]) for z in (lo[2], hi[2])])
    quads = [(0, 1, 3, 2, -1, 0, 0), (4, 6, 7, 5, 1, 0, 0), (0, 4, 5, 1, 0, -1, 0), (2, 3, 7, 6, 0, 1, 0),
             (0, 2, 6, 4, 0, 0, -1), (1, 5, 7, 3, 0, 0, 1)]
    out = []
    for a, b, d, e, *n in quads:
        for tri in ((a, b, d), (a, d, e)):
            out.append(np.concatenate([c[tri[0]], c[tri[1]], c[tri[2]], n]))
    return np.array(out, dtype=np.float64)


def shapes():
    for d in [(5, 31, 33), (4, 32, 64), (3, 30, 63), (3, 66, 29), (6, 34, 62)]:
        yield box((-0.37, -0.41, -0.43), (d[0] - 0.61, d[1] - 0.57, d[2] - 0.53)), d     # fluid on every face
        yield box((0.6, 0.7, 0.8), (d[0] - 1.3, d[1] - 1.4, d[2] - 1.6)), d              # one cell inside
    for axis, d in [(1, (15, 65, 35)), (2, (35, 15, 65))]:
        yield synth_cylinder(6.2, 61.0, 24, axis, ((d[0] - 1) / 2.0, (d[1] - 1) / 2.0, (d[2] - 1) / 2.0)), d
    yield np.concatenate([box((0.3, 0.3, 0.3), (7.7, 31.5, 31.5)), box((0.3, 32.6, 32.6), (7.7, 40.2, 63.4))]), (9, 44, 66)


HEADER = 88          # LBMCKPT2: the plane-major populations follow


def populations(path, dtype, Q):
    raw = np.fromfile(path, dtype=np.uint8)
    return raw, raw[HEADER:].view(dtype).reshape(Q, -1)


def stream_ref(flags, fstar, never):
    """Post-streaming, post-bounce-back populations of the fluid points, x-major, from f* of the fluid points."""
    m = LatticeModel(19)
    pad = np.full((19,) + tuple(n + 2 for n in flags.shape), np.nan)
    inner = pad[:, 1:-1, 1:-1, 1:-1]
    inner[:, flags] = fstar
    out = np.empty_like(fstar)
    for q in range(19):
        src = np.roll(pad[q], tuple(int(v) for v in m.c[q]), axis=(0, 1, 2))[1:-1, 1:-1, 1:-1][flags]
        back = fstar[m.opp[q]] if q != never else np.full(fstar.shape[1], m.w[q])
        out[q] = np.where(np.isnan(src), back, src)
    return out


@pytest.mark.parametrize("case", range(13))
@pytest.mark.parametrize("run_axis", [1, 2])
def test_lattice_on_word_edges(oracle_mod, tmp_path, case, run_axis):
    O = oracle_mod
    tris, dims = list(shapes())[case]
    geom = Geometry(tris, 1.0, grid=((0.0, 0.0, 0.0), dims))
    geo = O.geometry(tris, 1.0, ((0.0, 0.0, 0.0), dims), [])
    flags = geo["flags"].astype(bool).reshape(dims)
    assert np.array_equal(geom.flags().astype(bool), flags) and flags.any()
    assert np.array_equal(geom.boundaryPoints, geo["bidx"])
    rng = np.random.default_rng(case)
    path = str(tmp_path / "s.ckpt")

    sim = Simulation(geom, 0.9, (), precision="f64", pattern="pull", run_axis=run_axis)
    assert np.array_equal(sim.nodes(), np.flatnonzero(flags.ravel()))
    sim.checkpoint(path)
    raw, f = populations(path, np.float64, 19)
    f[:] = np.arange(f.shape[1])                     # every population of node id is id: the rest one never moves
    raw.tofile(path)
    sim.restart(path)
    ids = sim.fields(rho=False, u=False)[0][:, 18].astype(np.int64)
    assert len(np.unique(ids)) == len(ids)
    f[:] = LatticeModel(19).w[:, None] * rng.uniform(0.8, 1.2, f.shape)
    raw.tofile(path)
    sim.restart(path)
    got = sim.fields(rho=False, u=False)[0].T
    assert np.array_equal(got, stream_ref(flags, f[:, ids], LatticeModel(19).opp[0]))

    # (every missing population bounces back: the paired even launch relies on the odd one before it for the others)
    out = []
    for npl, ps in ((1, 0), (2, 8), (2, 16), (2, 32)):
        s = Simulation(geom, 0.9, (), precision="f32", pattern="aa", run_axis=run_axis, nodes_per_lane=npl, staging=1,
                       piece_slots=ps, corrections=1)
        if npl == 1:
            s.checkpoint(path)
            raw, f = populations(path, np.float32, 19)
            f[:] = LatticeModel(19).w[:, None].astype(np.float32) * rng.uniform(0.99, 1.01, f.shape).astype(np.float32)
            raw.tofile(path)
        s.restart(path)
        s.step(4)
        out.append(s.fields(rho=False, u=False)[0])
    assert np.array_equal(out[1], out[2]) and np.array_equal(out[1], out[3])
    assert np.linalg.norm(out[1] - out[0]) <= 1e-6 * np.linalg.norm(out[0])
