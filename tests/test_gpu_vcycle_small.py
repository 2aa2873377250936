"""The whole V-cycle of a small body in the cluster kernel, against level 0 in launches of its own: the same rows, lanes
and order, so the same frames bit for bit, at ragged sizes, both sides of the size rule, every precision and sweep count."""
import numpy as np
import pytest

import multigridsoftbody_b200 as mg

from .common import beam, capsule_path, mg_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,levels,sweeps,fused,precision,passes,whole", [
    ((1, 3, 1), 2, (2, 2), True, mg.PRECISION_FP32, 1, True),
    ((3, 11, 2), 2, (2, 2), True, mg.PRECISION_FP32, 1, True),
    ((4, 40, 4), 3, (2, 2), True, mg.PRECISION_FP32, 2, True),
    ((5, 37, 3), 3, (1, 1), True, mg.PRECISION_MIXED, 1, True),
    ((6, 20, 6), 4, (1, 0), True, mg.PRECISION_MIXED, 2, True),
    ((6, 20, 6), 3, (0, 0), False, mg.PRECISION_MIXED, 2, True),
    ((7, 33, 6), 4, (2, 3), False, mg.PRECISION_FP32, 2, True),
    ((7, 33, 6), 4, (3, 2), True, mg.PRECISION_MIXED, 2, True),
    ((6, 20, 6), 4, (0, 1), True, mg.PRECISION_FP32, 1, False),
    ((7, 35, 6), 4, (2, 2), True, mg.PRECISION_FP32, 1, False),
])
def test_same_bits_as_level0_launches(lib, dims, levels, sweeps, fused, precision, passes, whole):
    m, fixed = beam(*dims)
    p = mg_params(levels=levels, gravity=(0, -9.8, 0), precision=precision, pre_sweeps=sweeps[0], post_sweeps=sweeps[1],
                  refinement_passes=passes)
    path = capsule_path(4, start=(0.0, 0.0, 1.2))
    out, launches = [], []
    for own in (True, False):
        s = mg.Solver(m, p)
        s.set_fixed(fixed)
        if not own:
            s.set_kernel_shape(0, 0, 0)   # level 0 not fused
        s.set_fused_prolongation(fused)
        for a, b in path:
            s.set_capsule(a, b, 0.3)
            s.step()
        out.append(s.positions())
        launches.append(s.launches_per_frame())
        s.close()
    assert np.isfinite(out[0]).all() and np.abs(out[0] - m.positions).max() > 1e-4
    assert np.array_equal(out[0], out[1])
    assert (launches[0] < launches[1]) == whole
