"""The cluster kernel that keeps its operators in shared memory, against the one-CTA kernel: the same rows, lanes and
order, so the same frames bit for bit, at ragged sizes, every cluster size and sweep counts from none up."""
import numpy as np
import pytest

import multigridsoftbody_b200 as mg

from .common import beam, capsule_path, mg_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,levels,split,sweeps,fused,precision", [
    ((4, 40, 4), 3, 1, (2, 2), True, mg.PRECISION_FP32),
    ((5, 37, 3), 3, 1, (1, 1), True, mg.PRECISION_MIXED),
    ((7, 33, 6), 4, 1, (3, 2), True, mg.PRECISION_FP32),
    ((7, 33, 6), 4, 2, (2, 3), False, mg.PRECISION_FP32),
    ((3, 11, 2), 2, 1, (2, 2), True, mg.PRECISION_FP32),   # the coarsest level alone
    ((9, 50, 9), 4, 1, (0, 1), True, mg.PRECISION_FP32),
    ((9, 50, 9), 4, 2, (1, 0), True, mg.PRECISION_MIXED),
])
def test_same_bits_as_one_cta(lib, dims, levels, split, sweeps, fused, precision):
    m, fixed = beam(*dims)
    p = mg_params(levels=levels, gravity=(0, -9.8, 0), precision=precision, pre_sweeps=sweeps[0], post_sweeps=sweeps[1])
    path = capsule_path(4, start=(0.0, 0.0, 1.2))
    out = {}
    for cluster in (1, 2, 3, 8, 16, 0):   # 0: the solver's own choice
        s = mg.Solver(m, p)
        s.set_fixed(fixed)
        s.set_coarse_split(split)
        s.set_kernel_shape(cluster, 512 if cluster else 0, 0)
        s.set_fused_prolongation(fused)
        for a, b in path:
            s.set_capsule(a, b, 0.3)
            s.step()
        out[cluster] = s.positions()
        s.close()
    assert np.isfinite(out[1]).all() and np.abs(out[1] - m.positions).max() > 1e-4
    for cluster in (2, 3, 8, 16, 0):
        assert np.array_equal(out[1], out[cluster]), cluster
