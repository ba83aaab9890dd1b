"""Every gather shape gives the state of a thread per node bit for bit: groups
of 4, 8, 16 and 32 lanes (one node's terms added by one lane per sum), on a
mesh whose node counts leave a partly filled last warp on each level, and the
default choice on levels on both sides of its threshold.
"""
import ctypes

import numpy as np
import pytest

from conftest import oracle_backend
from flite3d_b200 import Mesh, Solver, default_controls, initial_state

pytestmark = pytest.mark.gpu

CASES = {
    "euler": dict(),
    "weighted": dict(useDissipationWeighting=1),
    "hllc2": dict(fluxType=4, HLLCFluxOrder=2, Automaticlipping=1, CFLNumber=1.0),
    "laminar": dict(ReynoldsNumber=500.0, CFLNumber=1.0, wallsAreIsentropic=1),
    "laminar_compact": dict(ReynoldsNumber=500.0, CFLNumber=1.0, viscosityScheme=2),
    "mixed": dict(precision=1),
}


def states(mesh, ctl, lanes, cycles=2):
    c = default_controls(**{**dict(ReynoldsNumber=0.0, fluxType=1, CFLNumber=2.0, multigridScheme=3,
                                   numberOfGridsToUse=mesh.nlevels), **ctl})
    s = Solver(c, mesh)
    for level in range(1, mesh.nlevels + 1):
        s.set_gather_lanes(level, lanes)
    s.set_state(initial_state(c, mesh, perturb_seed=5, amplitude=0.03))
    s.start()
    for it in range(1, cycles + 1):
        s.cycle(it)
    out = [s.get_state(level) for level in range(1, mesh.nlevels + 1)]
    s.close()
    return out


@pytest.mark.parametrize("name", list(CASES))
def test_group_shapes_match_a_thread_per_node(name):
    mesh = Mesh.bump_channel(17, 7, 6, 0.05, nlevels=3)
    want = states(mesh, CASES[name], 1)
    assert all(np.all(np.isfinite(u)) for u in want)
    # FLITE_MIXED sums FP32 increments in the same order in every shape
    for lanes in (4, 8, 16, 32, 0):
        for level, (a, b) in enumerate(zip(want, states(mesh, CASES[name], lanes)), 1):
            assert np.array_equal(a, b), (lanes, level)


@pytest.mark.parametrize("size", [(17, 7, 6), (40, 13, 13), (61, 19, 20), (75, 24, 25)])
def test_default_shape_matches_a_thread_per_node(size):
    mesh = Mesh.bump_channel(*size, 0.05, nlevels=3)
    for a, b in zip(states(mesh, CASES["laminar"], 1, 1), states(mesh, CASES["laminar"], 0, 1)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("ctl", [dict(rungeKuttaStages=5, CFLNumber=1.0), dict(multigridScheme=2), dict(multigridScheme=7),
                                 dict(numberOfRelaxationSteps=3), dict(boundaryTerm=2), dict(flowType=1, physicalTimeStep=0.2),
                                 dict(secondOrderDissipationFactor=0.0, fourthOrderDissipationFactor=0.0),
                                 dict(minimumDensity=1.0)],
                         ids=["five_stages", "w_cycle", "scheme7", "steps", "fv_boundary", "unsteady", "no_jst", "floored"])
@pytest.mark.parametrize("model", ["euler", "laminar"])
def test_passes_between_stages_match_the_restatement(model, ctl):
    """Stages that alternate the copies of the state, folded dissipation,
    boundary edges evaluated in the node pass, the floor left to the
    restriction, the branch of the restriction: bit for bit on every level."""
    mesh = Mesh.bump_channel(17, 7, 6, 0.05, nlevels=3)
    c = default_controls(**{**dict(ReynoldsNumber=0.0, fluxType=1, CFLNumber=2.0, multigridScheme=3,
                                   numberOfGridsToUse=3), **CASES[model], **ctl})
    u0 = initial_state(c, mesh, perturb_seed=5, amplitude=0.03)
    got = []
    for be in (None, oracle_backend()):
        s = Solver(c, mesh, backend=be)
        s.set_state(u0)
        s.start()
        for it in range(1, 4):
            s.cycle(it)
        got.append([s.get_state(level) for level in (1, 2, 3)] + [s.get_pressure()])
        s.close()
    for a, b in zip(*got):
        assert np.all(np.isfinite(b))
        assert np.array_equal(a, b)


def test_fine_nodes_without_a_parent_match_the_restatement():
    """Transfers where some fine nodes have no parent (the two-launch
    prolongation)."""
    mesh = Mesh.bump_channel(17, 7, 6, 0.05, nlevels=2)
    n = mesh.level(1).n_nodes
    parent = np.ctypeslib.as_array(ctypes.cast(mesh.level(2).parent, ctypes.POINTER(ctypes.c_int32)), (n,))
    parent[::37] = 0
    c = default_controls(ReynoldsNumber=0.0, fluxType=1, CFLNumber=1.0, multigridScheme=3, numberOfGridsToUse=2)
    got = []
    for be in (None, oracle_backend()):
        s = Solver(c, mesh, backend=be)
        s.set_state(initial_state(c, mesh, perturb_seed=5))
        s.start()
        for it in range(1, 3):
            s.cycle(it)
        got.append([s.get_state(level) for level in (1, 2)])
        s.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("size", [(46, 39, 40), (59, 51, 50)])
def test_residual_norms_of_large_levels_match_the_restatement(size):
    """Levels with more nodes than one pass of the norm's threads holds (77,080:
    a second node for some threads; 159,120: a second round).  Any order of a
    sum of n squares is within n eps of another, its root within half of that."""
    mesh = Mesh.bump_channel(*size, 0.05, nlevels=1)
    n = mesh.level(1).n_nodes
    assert n > 296 * 256
    c = default_controls(ReynoldsNumber=0.0, fluxType=1, CFLNumber=1.0, numberOfGridsToUse=1)
    got = []
    for be in (None, oracle_backend()):
        s = Solver(c, mesh, backend=be)
        s.set_state(initial_state(c, mesh, perturb_seed=5))
        s.start()
        s.cycle(1)
        got.append(s.residuals())
        s.close()
    (r, m, k), (r0, m0, k0) = got
    assert np.all(r0 > 0) and np.all(m0 > 0)
    np.testing.assert_allclose(r, r0, rtol=n * np.finfo(float).eps)
    assert np.array_equal(m, m0) and np.array_equal(k, k0)
