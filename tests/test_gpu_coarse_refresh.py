"""The coarse operator follows the step: after a step of another length (or a static
one) a handle's step is that of a handle that never took it, bit for bit and in as
many iterations."""
import numpy as np
import pytest

from sors_b200 import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,cells,precision", [("tet", (20, 4, 4), "fp64"), ("hex", (9, 9, 9), "mixed"),
                                                  ("tet", (27, 15, 21), "mixed")])
@pytest.mark.parametrize("first,then", [(0.0, 1e-4), (1e-2, 1e-4), (1e-4, 1e-2)])
def test_step_of_another_length(kind, cells, precision, first, then):
    from sors_b200 import py_sors as ps
    size = tuple(5e-3 * c for c in cells)
    X, T = meshes.hex_bar(*cells, size)
    if kind == "tet":
        T = meshes.kuhn_tet_elements(*cells)
        X = meshes.grid_nodes(*cells, size)
    mask, val = meshes.clamp_mask(X)
    v = np.where(mask == 1, 0.0, np.random.default_rng(2).uniform(-0.05, 0.05, X.size))
    out = []
    for dt in ((first, then), (then,)):
        s = ps.SimulationSettings()
        s.meshType = "Tetrahedron" if kind == "tet" else "Hexahedron"
        s.dt = dt[0]
        s.timeSteppingScheme = "backward_euler"
        s.precision = precision
        cls = ps.EnergyTet if kind == "tet" else ps.EnergyHex
        en = cls.from_arrays(X, T, s, np.array([0.0, 0.0, -1.0]), 0.0, density=1070.0, youngsModulus=1e4,
                             poissonsRatio=0.45, neumannBCmask=mask, neumannBCvalue=np.zeros(mask.size))
        sol = ps.Solver(s)
        for d in dt:
            en.set_initial_deformation(X.ravel())
            en.set_initial_velocity(v)
            q = sol.step(X.ravel(), en, None, d)
        out.append((q, sol.last_stats.pcg_iters))
    assert out[0][1] == out[1][1]
    assert np.array_equal(out[0][0], out[1][0])
