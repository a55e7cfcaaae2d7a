"""A bar compressed between its two ends, whose first Hessians are indefinite in the
coarse space as well: the correction is then left out, so that the default settings
take the step of block Jacobi alone (both stop at ||dx|| < 1e-9 m) in no more
iterations."""
import numpy as np
import pytest

from sors_b200 import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("comp,pert,dt", [(0.05, 2e-4, 1e-2), (0.2, 5e-4, 1e-2), (0.25, 2e-4, 2e-2), (0.3, 5e-4, 1e-2)])
def test_compressed_bar(precision, comp, pert, dt):
    from sors_b200 import py_sors as ps
    L = 0.08
    X, T = meshes.cantilever_tets(16, 4, 4, (L, 0.02, 0.02))
    ends = (np.abs(X[:, 0]) < 1e-12) | (np.abs(X[:, 0] - L) < 1e-12)
    mask = np.repeat(ends, 3).astype(np.int32)
    noise = pert * np.random.default_rng(0).standard_normal(X.size)
    q0 = (X * [1.0 - comp, 1.0, 1.0]).ravel() + noise * (1 - mask)
    out = []
    for two_level in ("auto", False):
        s = ps.SimulationSettings()
        s.meshType = "Tetrahedron"
        s.dt = dt
        s.timeSteppingScheme = "backward_euler"
        s.precision = precision
        s.twoLevelPreconditioner = two_level
        s.newtonPredictor = False
        en = ps.EnergyTet.from_arrays(X, T, s, np.zeros(3), 0.0, density=1000.0, youngsModulus=1e5, poissonsRatio=0.45,
                                      neumannBCmask=mask, neumannBCvalue=np.zeros(mask.size))
        en.set_initial_deformation(q0)
        sol = ps.Solver(s)
        out.append((sol.step(q0, en), sol.last_stats.pcg_iters))
    u = np.abs(out[1][0] - q0).max()
    assert np.abs(out[0][0] - out[1][0]).max() <= (1e-8 if precision == "fp64" else 1e-6 * u)
    assert out[0][1] <= out[1][1]
