"""A state that an evaluation rejects (inverted elements, NaN) leaves nothing
behind in the handle: what follows is what a handle that never saw it gives,
bit for bit and in as many iterations."""
import numpy as np
import pytest

from sors_b200 import meshes

pytestmark = pytest.mark.gpu

# N = 1,014 tet nodes in a cluster, 5,852 on a grid, 891 hex nodes: coarse correction on ("auto")
CASES = [("tet", (25, 12, 2), "fp64"), ("tet", (21, 13, 18), "mixed"), ("hex", (10, 8, 8), "fp64")]


def _energy(kind, cells, precision, predictor=True, energy="neohookean", v=0.0):
    from sors_b200 import py_sors as ps
    size = tuple(5e-3 * c for c in cells)
    if kind == "tet":
        X, T, E = meshes.jittered_block_tets(*cells, size, jitter=0.1, seed=1)
        E = 10.0 * E
    else:
        X, T = meshes.hex_bar(*cells, size)
        E = np.full(T.shape[0], 1e6)
    s = ps.SimulationSettings()
    s.meshType = "Tetrahedron" if kind == "tet" else "Hexahedron"
    s.dt = 1e-2
    s.timeSteppingScheme = "backward_euler"
    s.precision = precision
    s.newtonPredictor = predictor
    mask, val = meshes.clamp_mask(X)
    cls = ps.EnergyTet if kind == "tet" else ps.EnergyHex
    en = cls.from_arrays(X, T, s, np.array([0.0, 0.0, -9.81]), 0.0, density=1070.0, youngsModulus=E,
                         poissonsRatio=0.45, neumannBCmask=mask, neumannBCvalue=val, energy=energy)
    rng = np.random.default_rng(4)
    en.set_initial_velocity(np.where(mask == 1, 0.0, v * rng.uniform(-1.0, 1.0, X.size)))
    return X.ravel().copy(), en, ps.Solver(s)


def _step(q, en, sol):
    out = sol.step(q, en)
    return out, sol.last_stats.newton_iters, sol.last_stats.pcg_iters


@pytest.mark.parametrize("kind,cells,precision", CASES)
def test_inverted_prediction(kind, cells, precision):
    """q + dt v moves nodes by up to four cells, so the predicted start inverts
    elements and the step restarts from q: as with the prediction off."""
    got = []
    for predictor in (True, False):
        q, en, sol = _energy(kind, cells, precision, predictor, v=2.0)
        got.append(_step(q, en, sol))
    assert got[0][1:] == got[1][1:]
    assert np.array_equal(got[0][0], got[1][0])


@pytest.mark.parametrize("kind,cells,precision", CASES)
def test_nan_state(kind, cells, precision):
    """A stable Neo-Hookean step from NaN positions fails; the next valid step does not know of it."""
    q, en, sol = _energy(kind, cells, precision, energy="stableneohookean", v=0.01)
    ref = _step(q, en, sol)
    q, en, sol = _energy(kind, cells, precision, energy="stableneohookean", v=0.01)
    with pytest.raises(RuntimeError):
        sol.step(np.full_like(q, np.nan), en)
    got = _step(q, en, sol)
    assert got[1:] == ref[1:]
    assert np.array_equal(got[0], ref[0])


@pytest.mark.parametrize("kind,cells,precision", CASES)
def test_inverted_adjoint(kind, cells, precision):
    """An adjoint at a turned-over mesh fails; the next step does not know of it."""
    import ctypes as C

    from sors_b200 import _lib
    q, en, sol = _energy(kind, cells, precision, v=0.01)
    ref = _step(q, en, sol)
    q, en, sol = _energy(kind, cells, precision, v=0.01)
    dp = C.POINTER(C.c_double)
    bad = np.ascontiguousarray((q.reshape(-1, 3) * [1.0, 1.0, -1.0]).ravel())
    b, out = np.ones(q.size), np.zeros(q.size)
    with pytest.raises(RuntimeError):
        _lib.check(_lib.load().sors_adjoint_step(en.handle(), bad.ctypes.data_as(dp), 0.0, b.ctypes.data_as(dp), None,
                                                 None, 0, out.ctypes.data_as(dp), None, None, None, None, None))
    got = _step(q, en, sol)
    assert got[1:] == ref[1:]
    assert np.array_equal(got[0], ref[0])
