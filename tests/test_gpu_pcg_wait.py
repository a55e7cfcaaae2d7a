"""A wait between the blocks of the one-launch PCG that runs out (its limit set to a
single look, so that what other blocks send is never there in time) ends the solve
with an error; the handle's next step is that of a handle that never saw it."""
import ctypes as C
import time

import numpy as np
import pytest

from sors_b200 import meshes

pytestmark = pytest.mark.gpu


def _energy(cells, precision, two_level):
    from sors_b200 import py_sors as ps
    X, T, E = meshes.jittered_block_tets(*cells, tuple(5e-3 * c for c in cells), jitter=0.1, seed=3)
    s = ps.SimulationSettings()
    s.meshType = "Tetrahedron"
    s.dt = 2e-3
    s.timeSteppingScheme = "backward_euler"
    s.precision = precision
    s.twoLevelPreconditioner = two_level
    mask, val = meshes.clamp_mask(X)
    en = ps.EnergyTet.from_arrays(X, T, s, np.array([0.0, 0.0, -9.81]), 0.0, density=1070.0, youngsModulus=E,
                                  poissonsRatio=0.45, neumannBCmask=mask, neumannBCvalue=val)
    return X.ravel().copy(), en, ps.Solver(s)


def _run(cells, precision, two_level):
    from sors_b200 import _lib
    wait = _lib.load().sors_test_pcg_wait
    wait.restype, wait.argtypes = None, [C.c_void_p, C.c_uint64]
    q, en, sol = _energy(cells, precision, two_level)
    ref = sol.step(q, en), sol.last_stats.pcg_iters
    q, en, sol = _energy(cells, precision, two_level)
    wait(en.handle(), 0)
    t0 = time.perf_counter()
    for _ in range(2):
        with pytest.raises(RuntimeError, match="did not meet within the limit"):
            sol.step(q, en)
    assert time.perf_counter() - t0 < 2.0
    wait(en.handle(), 10**9)
    assert np.array_equal(sol.step(q, en), ref[0]) and sol.last_stats.pcg_iters == ref[1]


# N = 81, 525 and 1,014: three blocks (no coarse correction) and sixteen
@pytest.mark.parametrize("cells,precision", [((8, 2, 2), "mixed"), ((20, 4, 4), "fp64"), ((25, 12, 2), "mixed")])
@pytest.mark.parametrize("two_level", ["auto", False])
def test_cluster(cells, precision, two_level):
    _run(cells, precision, two_level)


# N = 4,225 and 9,856: eight and four lanes per row
@pytest.mark.parametrize("cells,precision", [((24, 12, 12), "fp64"), ((27, 15, 21), "mixed")])
@pytest.mark.parametrize("two_level", ["auto", False])
def test_grid(cells, precision, two_level):
    _run(cells, precision, two_level)


# 49k and 107k nodes: one and two aggregates per range
@pytest.mark.parametrize("cells,precision", [((40, 34, 33), "fp64"), ((57, 43, 41), "mixed")])
def test_streamed(cells, precision):
    _run(cells, precision, "auto")
