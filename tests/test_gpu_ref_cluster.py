"""The reference-faithful iterations of a body in one launch (one cluster for a small one, the whole grid for a larger
one) against a launch per step: the same body as one component of a larger mesh moves in the same bits, at ragged sizes,
one CTA's share of vertices and tets from none to many, and on the two-level schedule's coarse level with its triangle
contact."""
import numpy as np
import pytest

import multigridsoftbody_b200 as mg

from .common import beam

pytestmark = pytest.mark.gpu

GRID, LAUNCHES = (8, 50, 8), (16, 160, 16)   # company that makes a mesh too large for the cluster, for the grid


def _with_company(m, fixed, dims):
    """The mesh followed by a far larger one out of every tool's reach."""
    o, of = beam(*dims)
    far = o.positions + np.float32([100.0, 0.0, 0.0])
    n = len(m.positions)
    return (mg.TetMesh(np.concatenate([m.positions, far]), np.concatenate([m.tets, o.tets + n])),
            np.concatenate([fixed, of]))


def _spheres(frames, seed):
    rng = np.random.default_rng(seed)
    c = np.stack([np.linspace(1.5, 1.1, frames), np.full(frames, -3.0), np.zeros(frames)], 1)
    return (c + rng.normal(0.0, 0.01, c.shape)).astype(np.float32)


@pytest.mark.parametrize("dims,iterations", [
    ((1, 1, 1), 5), ((1, 3, 1), 2), ((2, 10, 2), 1), ((4, 14, 4), 20), ((3, 33, 5), 7), ((7, 31, 6), 20),
    ((8, 42, 8), 3), ((8, 42, 8), 1), ((11, 70, 13), 4),
])
def test_same_bits_as_launches(lib, dims, iterations):
    m, fixed = beam(*dims)
    n = len(m.positions)
    out, launches = [], []
    for mesh, fx in ((m, fixed), _with_company(m, fixed, GRID), _with_company(m, fixed, LAUNCHES)):
        s = mg.Solver(mesh, mg.default_params(mg.SOLVER_REFERENCE_JACOBI, iterations=iterations, gravity=(0.0, -9.8, 0.0)))
        s.set_fixed(fx)
        for c in _spheres(5, 3):
            s.set_spheres(c[None], [0.8])
            s.step()
        out.append((s.positions()[:n], s.velocities()[:n], s.contact_flags()[:n]))
        launches.append(s.launches_per_frame())
        s.close()
    assert launches == [1, 1, 1 + 2 * iterations]
    assert np.isfinite(out[0][0]).all() and np.abs(out[0][0] - m.positions).max() > 1e-5
    for a, b, c in zip(*out):
        assert np.array_equal(a, c) and np.array_equal(b, c)


@pytest.mark.parametrize("coarse,fine,iterations", [((2, 20, 2), (4, 40, 4), 9), ((4, 33, 4), (8, 66, 8), 4)])
def test_two_level_same_bits(lib, coarse, fine, iterations):
    (cm, cf), (fm, ff) = beam(*coarse), beam(*fine)
    out, hits = [], []
    for company in (None, GRID, LAUNCHES):
        c, cfx, f, ffx = cm, cf, fm, ff
        if company:
            c, cfx = _with_company(cm, cf, company)
            f, ffx = _with_company(fm, ff, company)
        t = mg.TwoLevel(c, f, mg.default_params(mg.SOLVER_REFERENCE_JACOBI, iterations=iterations))
        t.set_fixed(cfx, ffx)
        for q in _spheres(4, 5):
            t.set_spheres(q[None], [0.8])
            t.step()
        out.append((t.positions(0)[:len(fm.positions)], t.positions(1)[:len(cm.positions)]))
        hits.append(t.levels[1].contact_flags()[:len(cm.positions)])
        t.close()
    assert hits[0].sum() > 0 and np.array_equal(hits[0], hits[1]) and np.array_equal(hits[0], hits[2])
    for a, b, c in zip(*out):
        assert np.array_equal(a, c) and np.array_equal(b, c)
