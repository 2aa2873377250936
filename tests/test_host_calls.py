"""What the solvers' host code does when the runtime refuses a launch, and when set-up changes behind a captured frame:
the library over a stand-in for the CUDA runtime."""
import numpy as np
import pytest

import multigridsoftbody_b200 as mg
from multigridsoftbody_b200 import _lib as L
from multigridsoftbody_b200.learned import MLP

from .common import beam
from .host_only import ALLOCATED, CAPTURES, GRAPH_LAUNCHES, PINNED, UPLOADED, Host, build_host_only


@pytest.fixture(scope="module")
def host_library(tmp_path_factory):
    return Host(build_host_only(str(tmp_path_factory.mktemp("host"))))


@pytest.fixture
def host(host_library, monkeypatch):
    monkeypatch.setattr(L, "_lib", host_library.lib)
    host_library.reset()
    return host_library


def _two_level():
    (c, cf), (f, ff) = beam(2, 20, 2), beam(4, 40, 4)
    t = mg.TwoLevel(c, f, mg.default_params(mg.SOLVER_REFERENCE_JACOBI))
    t.set_fixed(cf, ff)
    return t


def test_refused_launch_fails_the_two_level_step(host):
    t = _two_level()
    host.refuse("k_ref_iterations")
    for _ in range(2):   # not kept as a frame without its iterations either
        with pytest.raises(mg.MgsbError, match="reference iterations launch failed"):
            t.step()
    assert host.count(GRAPH_LAUNCHES) == 0
    host.refuse("")
    host.reset()
    t.step()
    t.step()
    assert host.count(CAPTURES) == 1 and host.count(GRAPH_LAUNCHES) == 2 and len(host.launches("k_ref_iterations")) == 2
    t.close()


@pytest.mark.parametrize("level", [0, 1])
def test_level_set_up_by_its_own_handle_is_captured_again(host, level):
    (c, cf), (f, ff) = beam(2, 20, 2), beam(4, 40, 4)
    t = _two_level()
    t.step()
    own = t.levels[level]
    own.set_fixed((ff, cf)[level])
    own.normals()        # sets the level up again: the captured frame's buffers are gone
    t.step()
    assert host.count(CAPTURES) == 2
    own.set_launch_overlap(False)
    t.step()
    t.step()
    assert host.count(CAPTURES) == 3
    t.close()


@pytest.mark.parametrize("dims,levels,bodies", [((6, 60, 6), 3, 1), ((8, 80, 8), 3, 1), ((4, 40, 4), 3, 1), ((4, 40, 4), 3, 2)])
def test_autotune_offers_the_solvers_own_choice(host, dims, levels, bodies):
    m, fixed = beam(*dims)
    s = mg.Solver([m] * bodies, mg.default_params(mg.SOLVER_MULTIGRID, levels=levels))
    for b in range(bodies):
        s.set_fixed(fixed, body=b)
    s.step()
    own = host.launches("k_coarse_vcycle")[0]
    frame = s.launches_per_frame()
    host.reset()
    s.autotune(1)
    tried = host.launches("k_coarse_vcycle")
    assert own in tried and len(set(tried)) > 1
    # every candidate takes as long here: the own choice stays
    host.reset()
    s.step()
    assert host.launches("k_coarse_vcycle")[0] == own and s.launches_per_frame() == frame
    s.close()


def test_reference_plan_is_made_once_and_for_frames_only(host):
    m, fixed = beam(4, 40, 4)
    p = mg.default_params(mg.SOLVER_REFERENCE_JACOBI)
    s = mg.Solver(m, p)
    s.set_fixed(fixed)
    s.normals()
    s.energy()
    assert not host.launches("k_ref_image")
    s.step()
    assert len(host.launches("k_ref_image")) == 1 and len(host.launches("k_ref_iterations")) == 1
    for change in range(3):   # it depends on the mesh alone
        s.set_fixed(fixed if change else 1 - fixed)
        if change == 1:
            s.set_params(mg.default_params(mg.SOLVER_REFERENCE_JACOBI, iterations=7))
        s.step()
    assert len(host.launches("k_ref_image")) == 1 and len(host.launches("k_ref_iterations")) == 4
    s.close()
    host.reset()
    t = _two_level()
    assert not host.launches("k_ref_image")
    t.step()
    assert len(host.launches("k_ref_image")) == 2
    t.close()


@pytest.mark.parametrize("call", ["normals", "energy", "coarse_dense", "coarse_split", "precompute", "set_coarse_dense"])
def test_coarse_images_are_made_for_frames_only(host, call):
    m, fixed = beam(4, 40, 4)
    uploaded = []
    for first in (call, "step"):
        s = mg.Solver(m, mg.default_params(mg.SOLVER_MULTIGRID, levels=3))
        s.set_fixed(fixed)
        host.reset()
        {"set_coarse_dense": lambda: s.set_coarse_dense(False)}.get(first, getattr(s, first))()
        uploaded.append(host.count(UPLOADED))
        if first != "step":   # the rest is made by the first frame
            s.step()
            uploaded.append(host.count(UPLOADED))
        s.close()
    own, frame, whole = uploaded
    assert frame == whole and own < whole - 100_000


@pytest.mark.parametrize("solver,precision", [(mg.SOLVER_REFERENCE_JACOBI, 0), (mg.SOLVER_MULTIGRID, mg.PRECISION_FP32),
                                              (mg.SOLVER_MULTIGRID, mg.PRECISION_MIXED)])
def test_slots_are_placed_once(host, solver, precision):
    m, fixed = beam(4, 40, 4)
    s = mg.Solver(m, mg.default_params(solver, precision=precision))
    state = (5 * 16 + 32 * precision) * m.num_verts   # positions, predictions and earlier ones; FP64 ones of the mixed kind
    made = host.count(UPLOADED) - state
    host.reset()
    s.set_fixed(fixed)
    s.normals()
    # 16 bytes per tet of the reference kind; 8 + 8 of the multigrid kinds and more per vertex of a block
    assert 0 < host.count(UPLOADED) <= made - 16 * m.num_tets
    s.close()


@pytest.mark.parametrize("rows", [1, 128, 100_000])
def test_inference_pins_no_memory(host, rows):
    net = MLP(device=0, seed=0)
    y = net.forward(np.zeros((rows, 9), np.float32))
    assert y.shape == (rows, 3) and host.count(PINNED) == 0
    net.close()


@pytest.mark.parametrize("dims,levels", [((4, 40, 4), 3), ((9, 50, 9), 4)])
def test_blocks_of_shuffled_tets_are_compact(host, dims, levels):
    """The local step's shared memory grows with the vertices of its largest block."""
    m, fixed = beam(*dims)
    need = []
    for order in (np.arange(m.num_tets), np.random.default_rng(1).permutation(m.num_tets)):
        host.reset()
        s = mg.Solver([m, mg.TetMesh(m.positions, np.ascontiguousarray(m.tets[order]))],
                      mg.default_params(mg.SOLVER_MULTIGRID, levels=levels))
        for _ in range(2):
            s.step()
            s.set_fixed(fixed)
        launches = host.launches("k_mg_local")
        assert len({x[1:] for x in launches}) == 1
        need.append(launches[0][5])
        s.close()
    assert need[1] < 1.25 * need[0]


@pytest.mark.parametrize("dims,shuffled,one", [
    ((4, 40, 4), True, True), ((6, 40, 6), True, True), ((8, 49, 8), False, True), ((8, 49, 8), True, False),
    ((12, 112, 12), False, True), ((13, 120, 12), False, True), ((13, 130, 13), False, False), ((16, 160, 16), False, False),
])
def test_reference_bodies_in_one_launch(host, dims, shuffled, one):
    """Up to 1,792 tets in the fullest of 148 CTAs (1,752 at 22,022 vertices, 1,966 at 25,676), and windows of 3,072
    vertices (a shuffled body's are the whole of it)."""
    m, _ = beam(*dims)
    if shuffled:
        to = np.random.default_rng(3).permutation(m.num_verts).astype(np.int32)
        m = mg.TetMesh(np.ascontiguousarray(m.positions[np.argsort(to)]), np.ascontiguousarray(to[m.tets]))
    s = mg.Solver(m, mg.default_params(mg.SOLVER_REFERENCE_JACOBI))
    s.step()
    assert len(host.launches("k_ref_iterations")) == one and len(host.launches("k_ref_local")) == (0 if one else 20)
    assert len(host.launches("k_ref_image")) == one
    s.close()


@pytest.mark.parametrize("change", ["on", "split"])
def test_dense_operator_belongs_to_its_shape(host, change):
    """Residuals measured after the coarse shape changed, with no frame between: the operator is formed for it first."""
    m, fixed = beam(6, 40, 6)
    s = mg.Solver(m, mg.default_params(mg.SOLVER_MULTIGRID, levels=3))
    s.set_fixed(fixed)
    if change == "split":
        s.set_coarse_split(2)
        s.set_coarse_dense(True)
    s.step()
    if change == "on":
        s.set_coarse_dense(True)
    else:
        s.set_coarse_split(1)
    host.reset()
    s.vcycle_residuals(2)
    s.vcycle_residuals(1)
    order = [x[0] for x in host.launches("") if "k_op_init" in x[0] or "k_coarse_apply" in x[0]]
    assert len(order) == 4 and "k_op_init" in order[0] and all("k_coarse_apply" in x for x in order[1:])
    s.close()


def test_dense_operator_memory_is_for_its_users(host):
    m, _ = beam(6, 40, 6)
    allocated = []
    for dense in (False, True):
        host.reset()
        s = mg.Solver(m, mg.default_params(mg.SOLVER_MULTIGRID, levels=3))
        s.set_coarse_dense(dense)
        s.step()
        assert len(host.launches("k_op_init")) == dense and len(host.launches("k_coarse_apply")) == 10 * dense
        allocated.append(host.count(ALLOCATED))
        blocks = 16 * s.level_size(1)[0] ** 2
        s.close()
    assert allocated[1] - allocated[0] > 0.75 * blocks   # a plain solver has the cluster kernel's images instead
