"""Plans that are kept over set-ups: a solver whose masks, stiffness and iterations change between frames moves in the
bits of one that was made anew for each frame."""
import numpy as np
import pytest

import multigridsoftbody_b200 as mg

from .common import beam

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(3, 12, 3), (8, 42, 8), (16, 160, 16)])   # one cluster, the grid, launches
def test_reference_frames_over_set_ups(lib, dims):
    m, fixed = beam(*dims)
    half = (m.positions[:, 1] > 0).astype(np.uint8)
    steps = [dict(), dict(mask=half), dict(iterations=3), dict(iterations=0), dict(volume_stiffness=2000.0),
             dict(iterations=9, cheb_rho=0.9), dict(mask=fixed, dt=0.01)]
    params = dict(iterations=5, gravity=(0.0, -9.8, 0.0))
    make = lambda: mg.Solver(m, mg.default_params(mg.SOLVER_REFERENCE_JACOBI, **params))
    s, mask = make(), fixed
    s.set_fixed(mask)
    flags = np.zeros(len(m.positions), np.int32)
    x, v = m.positions, np.zeros_like(m.positions)
    for k, change in enumerate(steps):
        mask = change.pop("mask", mask)
        params.update(change)
        if change:
            s.set_params(**change)
        s.set_fixed(mask)
        fresh = make()
        fresh.set_fixed(mask)
        fresh.set_state(x, v)
        for q in (s, fresh):
            q.set_spheres([[1.5 - 0.03 * k, -3.0, 0.0]], [0.8])
            q.step()
        x, v = s.positions(), s.velocities()
        assert np.array_equal(x, fresh.positions()) and np.array_equal(v, fresh.velocities()), (k, change)
        if params["iterations"]:   # a frame without iterations finds no contact: the flags stay the last ones
            flags = fresh.contact_flags()
        assert np.array_equal(s.contact_flags(), flags)
        fresh.close()
    s.close()


@pytest.mark.parametrize("precision", [mg.PRECISION_FP32, mg.PRECISION_MIXED])
@pytest.mark.parametrize("dims", [[(3, 12, 3)], [(7, 35, 6)], [(2, 5, 2), (4, 19, 3)]])   # whole V-cycle, coarse part, batch
def test_multigrid_frames_over_set_ups(lib, dims, precision):
    bodies = [beam(*d) for d in dims]
    steps = [dict(), dict(flip=True), dict(iterations=3), dict(youngs=4e4), dict(iterations=6, pre_sweeps=1, dt=0.01)]
    params = dict(iterations=4, levels=3, gravity=(0.0, -9.8, 0.0), precision=precision)
    make = lambda: mg.Solver([m for m, _ in bodies], mg.default_params(mg.SOLVER_MULTIGRID, **params))
    s, flip, youngs = make(), False, None
    state = [(m.positions, np.zeros_like(m.positions)) for m, _ in bodies]
    for change in steps:
        flip, youngs = change.pop("flip", flip), change.pop("youngs", youngs)
        params.update(change)
        if change:
            s.set_params(**change)
        fresh = make()
        for q in (s, fresh):
            for b, (m, fixed) in enumerate(bodies):
                q.set_fixed(1 - fixed if flip else fixed, body=b)
                if youngs:
                    q.set_material(youngs, 0.3, body=b)
                q.set_state(*state[b], body=b)
            q.step(2)
        state = [(s.positions(b), s.velocities(b)) for b in range(len(bodies))]
        for b, (x, v) in enumerate(state):
            assert np.isfinite(x).all() and np.array_equal(x, fresh.positions(b)) and np.array_equal(v, fresh.velocities(b))
        fresh.close()
    s.close()


@pytest.mark.parametrize("dims,levels", [((6, 40, 6), 3), ((8, 80, 8), 4)])
def test_residuals_after_a_change_of_coarse_shape(lib, dims, levels):
    """No frame between: the dense operator is formed for the new shape, the same V-cycle up to rounding (496 products
    of FP32 at most: 3e-5 of the first residual)."""
    m, fixed = beam(*dims)
    s = mg.Solver(m, mg.default_params(mg.SOLVER_MULTIGRID, levels=levels))
    s.set_fixed(fixed)
    s.step(2)
    want = s.vcycle_residuals(3)
    for split, dense in ((levels - 1, True), (levels - 2, True), (levels - 2, False), (levels - 1, True)):
        s.set_coarse_split(split)
        s.set_coarse_dense(dense)
        got = s.vcycle_residuals(3)
        assert np.abs(got - want).max() < 1e-4 * want[0], (split, dense, got, want)
    s.close()
