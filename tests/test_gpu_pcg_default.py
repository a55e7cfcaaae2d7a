"""The one-launch PCG with its coarse correction as the default settings run it, in
every shape of its kernels, and the calls that a plain converging step does not
make (constraint projection, negative curvature, a solve that is skipped), in
every form: cluster, grid, streamed and launch per kernel.  The smaller meshes
take a later form by having the earlier ones' plans refused."""
import ctypes as C

import numpy as np
import pytest

from sors_b200 import meshes
from tests.helpers import contact_pair
from tests.test_gpu_pcg_resident import _large

pytestmark = pytest.mark.gpu

# grid: eight, four and two lanes per row, rows beyond one per group, hexes (eight and four
# lanes), a handle capped to 18 blocks; cluster: four lanes
SHAPES = [("tet", (24, 12, 12), "fp64", 0), ("tet", (21, 22, 23), "fp64", 0), ("tet", (27, 15, 21), "mixed", 0),
          ("tet", (30, 26, 24), "mixed", 0), ("tet", (33, 33, 33), "mixed", 0), ("tet", (26, 26, 26), "fp64", 0),
          ("hex", (40, 8, 8), "fp64", 0), ("hex", (23, 23, 23), "fp64", 0), ("hex", (25, 22, 22), "mixed", 0),
          ("tet", (19, 20, 20), "mixed", 148), ("tet", (18, 16, 16), "mixed", 8), ("tet", (14, 12, 12), "mixed", 0)]


@pytest.mark.parametrize("kind,cells,precision,cap", SHAPES)
@pytest.mark.parametrize("two_level", ["auto", False])
def test_shapes_match_minres(kind, cells, precision, cap, two_level):
    """A step against MINRES's separate kernels in FP64: both stop at ||dx|| < 1e-9 m;
    mixed precision is held to 1e-6 of the displacement."""
    from sors_b200 import py_sors as ps
    out = []
    for solver, prec, tl in (("minres", "fp64", False), ("pcg", precision, two_level)):
        s = ps.SimulationSettings()
        s.meshType = "Tetrahedron" if kind == "tet" else "Hexahedron"
        s.dt = 2e-3
        s.timeSteppingScheme = "backward_euler"
        s.precision = prec
        s.linearSolver = solver
        s.twoLevelPreconditioner = tl
        s.maxBlocksPerKernel = cap
        X, en, _ = _large(kind, cells, s)
        out.append(ps.Solver(s).step(X.ravel(), en))
    tol = 1e-8 if precision == "fp64" else 1e-6 * np.abs(out[0] - X.ravel()).max()
    assert np.abs(out[1] - out[0]).max() <= tol


class _refuse:
    """The next `n` plans of the one-launch PCG find no room."""

    def __init__(self, n):
        self.n = n

    def __enter__(self):
        from sors_b200 import _lib
        _lib.load().sors_test_deny(self.n, 0)

    def __exit__(self, *a):
        from sors_b200 import _lib
        _lib.load().sors_test_deny(0, 0)


def _form(en):
    from sors_b200 import _lib
    return _lib.load().sors_test_pcg_form(en.handle())


# plans refused, form then
FORMS = [(0, 1), (1, 2), (2, 3), (3, 0)]


def _contact(precision, two_level, refused):
    X = meshes.grid_nodes(10, 6, 6, (0.025, 0.015, 0.015)) + np.array([0.0, 0.0, 0.0003])
    en, sol, _, _ = contact_pair(X, meshes.kuhn_tet_elements(10, 6, 6), planes=([[0, 0, 0]], [[0, 0, 1.0]]), dt=2e-3,
                                 precision=precision, two_level=two_level)
    x = X.ravel().copy()
    with _refuse(refused):
        for _ in range(8):
            x = sol.step(x, en)
    return X.ravel(), x, en


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("refused,form", FORMS)
def test_contact_in_every_form(precision, refused, form):
    """SQP steps onto a plane (projected solves) give those of block Jacobi in launches per
    kernel: to 1e-9 m in FP64 as the two-level contact test, 1e-6 of the displacement in mixed."""
    X, a, en = _contact(precision, True, refused)
    assert _form(en) == form
    _, b, ref = _contact(precision, False, 3)
    assert _form(ref) == 0
    assert en.active_contacts() == ref.active_contacts() > 0
    assert np.abs(a - b).max() <= (1e-9 if precision == "fp64" else 1e-6 * np.abs(b - X).max())


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("refused,form", FORMS)
def test_negative_curvature_in_every_form(precision, refused, form):
    """A bar compressed by 15 % between its ends, whose first Newton matrices are indefinite: a solve
    reports the direction it met (p'Hp < 0) and the step converges on the projected matrix.  The gradient
    left is below dx_tol (1e-9 m) times a node's stiffness sum (under 1e5 N/m), against newtons at the start."""
    from sors_b200 import _lib
    from sors_b200 import py_sors as ps
    L = 0.08
    X, T = meshes.cantilever_tets(16, 4, 4, (L, 0.02, 0.02))
    ends = (np.abs(X[:, 0]) < 1e-12) | (np.abs(X[:, 0] - L) < 1e-12)
    mask = np.repeat(ends, 3).astype(np.int32)
    q0 = (X * [0.85, 1.0, 1.0]).ravel() + 5e-4 * np.random.default_rng(0).standard_normal(X.size) * (1 - mask)
    s = ps.SimulationSettings()
    s.meshType = "Tetrahedron"
    s.dt = 1e-2
    s.timeSteppingScheme = "backward_euler"
    s.precision = precision
    s.twoLevelPreconditioner = True
    s.newtonPredictor = False

    def energy():
        en = ps.EnergyTet.from_arrays(X, T, s, np.zeros(3), 0.0, density=1000.0, youngsModulus=1e5, poissonsRatio=0.45,
                                      neumannBCmask=mask, neumannBCvalue=np.zeros(mask.size))
        en.set_initial_deformation(q0)
        return en

    en = energy()
    with _refuse(refused):
        q = ps.Solver(s).step(q0, en)
    assert _form(en) == form
    rq, n = C.c_double(), C.c_int32()
    assert _lib.load().sors_last_step_curvature(en.handle(), C.byref(rq), C.byref(n)) == 0
    assert n.value > 0 and rq.value < 0.0
    assert np.abs(energy().compute_gradient(q, s.dt)).max() < 1e-4


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("refused,form", FORMS)
def test_skipped_solve_in_every_form(precision, refused, form):
    """A step at rest ends at the gradient: its solve is skipped on the device, and the next step
    is that of a handle that never took it (both stop at ||dx|| < 1e-9 m)."""
    from sors_b200 import py_sors as ps
    X, T, E = meshes.jittered_block_tets(12, 6, 6, (0.06, 0.03, 0.03), jitter=0.1, seed=3)
    s = ps.SimulationSettings()
    s.meshType = "Tetrahedron"
    s.dt = 2e-3
    s.timeSteppingScheme = "backward_euler"
    s.precision = precision
    s.twoLevelPreconditioner = True
    s.newtonResidualTol = 1e-9
    mask, val = meshes.clamp_mask(X)
    v = np.where(mask == 1, 0.0, np.random.default_rng(2).uniform(-0.1, 0.1, X.size))
    out = []
    for rest in (True, False):
        en = ps.EnergyTet.from_arrays(X, T, s, np.zeros(3), 0.0, density=1070.0, youngsModulus=E, poissonsRatio=0.45,
                                      neumannBCmask=mask, neumannBCvalue=val)
        sol = ps.Solver(s)
        with _refuse(refused if rest else 3):
            if rest:
                assert np.array_equal(sol.step(X.ravel(), en), X.ravel()) and sol.last_stats.pcg_iters == 0
            en.set_initial_deformation(X.ravel())
            en.set_initial_velocity(v)
            out.append(sol.step(X.ravel(), en))
        assert _form(en) == (form if rest else 0)
    assert np.abs(out[0] - out[1]).max() <= (1e-8 if precision == "fp64" else 1e-6 * np.abs(out[1] - X.ravel()).max())
