"""The two-level schedule without a coarse mask: a body with no fixed vertex, and one whose mask is set on the fine
level alone.  Frames and coarse contact flags against the FP64 oracle."""
import numpy as np
import pytest

import multigridsoftbody_b200 as mg
from oracle.binding import OracleTwoLevel

from .golden.make_golden import mg2_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fine_mask", [False, True])
@pytest.mark.parametrize("frames", [1, 6])
def test_coarse_contact_without_a_coarse_mask(lib, oracle_built, fine_mask, frames):
    coarse, fine, _, ff = mg2_scene()
    p = mg.default_params(mg.SOLVER_REFERENCE_JACOBI, gravity=(0.0, 0.0, 0.0))
    t, o = mg.TwoLevel(coarse, fine, p), OracleTwoLevel(coarse, fine, p)
    if fine_mask:
        t.set_fixed(None, ff)
        o.levels[0].set_fixed(ff)
    for f in range(frames):
        center = [[1.45 - 0.02 * f, -3.0, 0.2]]
        for x in (t, o):
            x.set_spheres(center, [0.8])
            x.step()
    diag = fine.bbox_diagonal()
    flags = t.levels[1].contact_flags()
    assert flags.sum() > 0 and np.array_equal(flags, o.contact_flags(1))
    for level in (0, 1):
        # reference-kind tolerance: FP32 vs FP64 of an iteration that amplifies perturbations
        assert np.abs(t.positions(level) - o.positions(level)).max() < 5e-5 * diag, level
    t.close()
