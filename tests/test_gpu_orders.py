"""Bodies whose vertices or tets come in another order than a voxel mesher's: the blocks of tets, the windows and the
images of the one-launch kernels, and the kernels that take over where a numbering reaches too far."""
import numpy as np
import pytest

import multigridsoftbody_b200 as mg
from oracle.binding import Oracle, OracleTwoLevel

from .common import beam, capsule_path, mg_params
from .test_gpu_ref_cluster import LAUNCHES, _spheres, _with_company

pytestmark = pytest.mark.gpu

ORDERS = ["vertices", "tets", "both", "reversed", "interleaved"]


def _reordered(dims, order):
    """A beam with its vertices, its tets or both shuffled, turned round, or its two halves' vertices taken in turn."""
    m, fixed = beam(*dims)
    rng = np.random.default_rng(len(order))
    n, T = len(m.positions), len(m.tets)
    v = {"vertices": rng.permutation(n), "both": rng.permutation(n), "reversed": np.arange(n)[::-1],
         "interleaved": np.argsort(np.arange(n) % ((n + 1) // 2), kind="stable")}.get(order, np.arange(n))
    t = {"tets": rng.permutation(T), "both": rng.permutation(T), "reversed": np.arange(T)[::-1]}.get(order, np.arange(T))
    place = np.empty(n, np.int32)
    place[v] = np.arange(n, dtype=np.int32)
    return (mg.TetMesh(np.ascontiguousarray(m.positions[v]), np.ascontiguousarray(place[m.tets[t]])),
            np.ascontiguousarray(fixed[v]))


@pytest.mark.parametrize("precision", [mg.PRECISION_FP32, mg.PRECISION_MIXED])
@pytest.mark.parametrize("order", ORDERS)
@pytest.mark.parametrize("dims,levels", [((4, 30, 4), 3), ((8, 48, 8), 4)])   # whole V-cycle in the cluster, coarse part
def test_multigrid_frames_match_oracle(lib, oracle_built, dims, levels, order, precision):
    m, fixed = _reordered(dims, order)
    p = mg_params(levels=levels, gravity=(0.0, 0.0, 0.0), precision=precision,
                  refinement_passes=2 if precision == mg.PRECISION_MIXED else 1)
    s, o = mg.Solver(m, p), Oracle(m, p)
    contacts = 0
    for q in (s, o):
        q.set_fixed(fixed)
    for a, b in capsule_path(4, start=(0.0, 0.0, 1.25)):
        for q in (s, o):
            q.set_capsule(a, b, 0.3)
            q.step()
        assert np.array_equal(s.contact_flags(), o.contact_flags())
        contacts += int(o.contact_flags().sum())
    x = s.positions_f64() if precision == mg.PRECISION_MIXED else s.positions()
    assert contacts > 0 and np.abs(x - o.positions()).max() < 1e-5 * m.bbox_diagonal()
    s.close()


@pytest.mark.parametrize("order", ORDERS)
@pytest.mark.parametrize("dims,levels,precision", [
    ((4, 30, 4), 3, mg.PRECISION_FP32), ((7, 31, 6), 4, mg.PRECISION_MIXED), ((9, 50, 9), 4, mg.PRECISION_FP32),
    ((12, 100, 12), 4, mg.PRECISION_FP32),   # 1,656 rows on level 1: over 2 to 8 CTAs the images do not fit
])
def test_same_bits_in_every_coarse_kernel(lib, order, dims, levels, precision):
    m, fixed = _reordered(dims, order)
    p = mg_params(levels=levels, gravity=(0, -9.8, 0), precision=precision, iterations=4)
    path = capsule_path(2, start=(0.0, 0.0, 1.2))
    out = []
    for cluster in (1, 2, 5, 8, 16, 0):   # 1: one CTA; 0: the solver's own choice
        s = mg.Solver(m, p)
        s.set_fixed(fixed)
        if cluster or len(m.positions) > 2000:   # smaller ones: the whole V-cycle by the solver's own choice
            s.set_coarse_split(1)
        if cluster:
            s.set_kernel_shape(cluster, 512, 0)
        for a, b in path:
            s.set_capsule(a, b, 0.3)
            s.step()
        out.append(s.positions())
        s.close()
    assert np.isfinite(out[0]).all() and np.abs(out[0] - m.positions).max() > 1e-5
    for x in out[1:]:
        assert np.array_equal(x, out[0])


@pytest.mark.parametrize("order", ORDERS)
@pytest.mark.parametrize("dims,iterations", [((1, 3, 1), 3), ((4, 14, 4), 20), ((5, 30, 5), 6), ((8, 42, 8), 5),
                                             ((12, 60, 12), 3)])
def test_reference_same_bits_as_launches(lib, order, dims, iterations):
    m, fixed = _reordered(dims, order)
    n, out = len(m.positions), []
    for mesh, fx in ((m, fixed), _with_company(m, fixed, LAUNCHES)):
        s = mg.Solver(mesh, mg.default_params(mg.SOLVER_REFERENCE_JACOBI, iterations=iterations, gravity=(0.0, -9.8, 0.0)))
        s.set_fixed(fx)
        for c in _spheres(4, 3):
            s.set_spheres(c[None], [0.8])
            s.step()
        out.append((s.positions()[:n], s.velocities()[:n], s.contact_flags()[:n]))
        s.close()
    assert np.isfinite(out[0][0]).all() and np.abs(out[0][0] - m.positions).max() > 1e-5
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("order", ORDERS)
def test_two_level_frames_match_oracle(lib, oracle_built, order):
    (cm, cf), (fm, ff) = _reordered((2, 12, 2), order), _reordered((4, 24, 4), order)
    p = mg.default_params(mg.SOLVER_REFERENCE_JACOBI, iterations=8)
    t, o = mg.TwoLevel(cm, fm, p), OracleTwoLevel(cm, fm, p)
    for q in (t, o):
        q.set_fixed(cf, ff)
    for f in range(4):
        for q in (t, o):
            q.set_spheres([[1.45 - 0.02 * f, -3.0, 0.2]], [0.8])
            q.step()
    flags = t.levels[1].contact_flags()
    assert flags.sum() > 0 and np.array_equal(flags, o.contact_flags(1))
    for level in (0, 1):
        assert np.abs(t.positions(level) - o.positions(level)).max() < 5e-5 * fm.bbox_diagonal(), level
    t.close()


@pytest.mark.parametrize("order", ["tets", "both"])
def test_material_follows_its_tet(lib, order):
    """Tets that the plan takes in another order keep their material through set-ups: energies and frames are those of
    the mesh in its own order, up to the order of sums."""
    m, fixed = beam(6, 30, 6)
    r, rfixed = _reordered((6, 30, 6), order)
    at = {tuple(p): i for i, p in enumerate(m.positions)}
    back = np.array([at[tuple(p)] for p in r.positions])            # a vertex's number in the mesh's own order
    young = {tuple(sorted(t)): 5e4 * (1 + k % 7) for k, t in enumerate(m.tets)}
    stretched = m.positions * np.float32([1.02, 1.05, 0.97])
    out, energies = [], []
    for mesh, fx, ids in ((m, fixed, np.arange(len(back))), (r, rfixed, back)):
        e = np.array([young[tuple(sorted(ids[t]))] for t in mesh.tets], np.float32)
        s = mg.Solver(mesh, mg_params(levels=3, gravity=(0.0, 0.0, 0.0)))
        for _ in range(2):   # the second set-up takes the order from the first
            s.set_fixed(fx)
            s.set_material(e, 0.3)
            s.set_state(stretched[ids], np.zeros_like(stretched))
            energies.append(s.energy())
            s.step()
        x = np.empty_like(m.positions)
        x[ids] = s.positions()
        out.append(x)
        s.close()
    for k in (0, 1):   # kinetic energy is measured from the frame before: pass by pass
        np.testing.assert_allclose(energies[2 + k][:4], energies[k][:4], rtol=1e-6)
    assert np.abs(out[0] - stretched).max() > 1e-3 and np.abs(out[1] - out[0]).max() < 1e-5 * m.bbox_diagonal()
