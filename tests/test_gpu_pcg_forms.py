"""Meshes that the first form of the one-launch PCG refuses take the next one:
a step's solves are launches of their own, not launches per PCG iteration, and the
step is the one that MINRES's separate kernels give (both stop at ||dx|| < 1e-9 m)."""
import numpy as np
import pytest

from sors_b200 import meshes

pytestmark = pytest.mark.gpu


def _step(X, T, E, solver, deny=0, threads=0):
    from sors_b200 import _lib
    from sors_b200 import py_sors as ps
    s = ps.SimulationSettings()
    s.meshType = "Tetrahedron" if T.shape[1] == 4 else "Hexahedron"
    s.dt = 2e-3
    s.timeSteppingScheme = "backward_euler"
    s.linearSolver = solver
    mask, val = meshes.clamp_mask(X)
    used = np.zeros(X.shape[0], bool)
    used[T.ravel()] = True
    mask = np.where(np.repeat(used, 3), mask, 1)
    cls = ps.EnergyTet if T.shape[1] == 4 else ps.EnergyHex
    en = cls.from_arrays(X, T, s, np.array([0.0, 0.0, -9.81]), 0.0, density=1070.0, youngsModulus=E,
                         poissonsRatio=0.45, neumannBCmask=mask, neumannBCvalue=np.zeros(X.size))
    v = np.random.default_rng(2).uniform(-0.1, 0.1, X.size)
    en.set_initial_velocity(np.where(mask == 1, 0.0, v))
    sol = ps.Solver(s)
    n0 = _lib.load().sors_kernel_launch_count()
    _lib.load().sors_test_deny(deny, threads)
    try:
        q = sol.step(X.ravel(), en)
    finally:
        _lib.load().sors_test_deny(0, 0)
    return q, _lib.load().sors_kernel_launch_count() - n0, sol.last_stats


def test_range_with_too_many_rows():
    """600 nodes without elements, each a row of one block, before a cube of 2,197 nodes:
    the cluster's first range would have more rows than a block takes, the grid's has not."""
    X, T, E = meshes.jittered_block_tets(12, 12, 12, (0.06,) * 3, jitter=0.1, seed=5)
    far = np.random.default_rng(1).uniform(0.0, 0.06, (600, 3))
    X, T = np.concatenate([far, X]), T + 600
    q, launches, st = _step(X, T, E, "pcg")
    assert launches < st.pcg_iters
    assert np.abs(q - _step(X, T, E, "minres")[0]).max() <= 1e-8


@pytest.mark.parametrize("cells,deny,one_launch", [((20, 21, 21), 1, True), ((20, 21, 21), 2, False),
                                                   ((7, 8, 6), 1, True), ((7, 8, 6), 3, False)])
def test_no_room_for_the_plan(cells, deny, one_launch):
    """The plan's allocation fails on the device, once or for every form: the step is made all the same."""
    X, T, E = meshes.jittered_block_tets(*cells, tuple(5e-3 * c for c in cells), jitter=0.1, seed=5)
    q, launches, st = _step(X, T, E, "pcg", deny)
    assert (launches < st.pcg_iters) == one_launch
    assert np.abs(q - _step(X, T, E, "minres")[0]).max() <= 1e-8


@pytest.mark.parametrize("threads", [1, 100])
def test_no_threads_for_the_plan(threads):
    """The host starts some or none of the streamed plan's threads: the plan is made on those that there are."""
    X, T, E = meshes.jittered_block_tets(20, 21, 21, (0.1, 0.105, 0.105), jitter=0.1, seed=5)
    a, launches, st = _step(X, T, E, "pcg", 1, threads)
    assert launches < st.pcg_iters
    assert np.array_equal(a, _step(X, T, E, "pcg", 1)[0])
