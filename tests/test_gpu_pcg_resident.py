"""The one-launch PCG (matrix resident on the SMs) at the sizes where its plan
changes: a single block, a partly filled cluster, ranges with rows beyond the
register-held ones, the grid form with eight, four and two lanes per row, and
hex rows.  The step is compared with Newton's method on the host: gradient and
Hessian from the Energy calls, each system solved by SciPy's CG to 1e-13.
Both stop at ||dx|| < 1e-9 m, so 1e-8 m separates a wrong solve from a right one
in FP64; mixed precision is held to 1e-6 of the displacement, as elsewhere."""
import numpy as np
import pytest

from sors_b200 import meshes

pytestmark = pytest.mark.gpu

# (kind, cells, precision): N = 8 | 81 | 1,014 | 3,375 | 4,800 | 8,470 | 2,205 hex
CASES = [("tet", (1, 1, 1), "fp64"), ("tet", (8, 2, 2), "mixed"), ("tet", (25, 12, 2), "fp64"),
         ("tet", (14, 14, 14), "fp64"), ("tet", (14, 15, 19), "fp64"), ("tet", (10, 34, 21), "mixed"),
         ("tet", (10, 34, 21), "fp64"), ("hex", (20, 6, 14), "fp64"), ("hex", (3, 2, 2), "mixed")]


def _energy(kind, cells, precision, method="minimize_newton"):
    from sors_b200 import py_sors as ps
    size = tuple(5e-3 * c for c in cells)
    rng = np.random.default_rng(sum(cells))
    if kind == "tet":
        X, T, E = meshes.jittered_block_tets(*cells, size, jitter=0.1, seed=sum(cells))
    else:
        X, T = meshes.hex_bar(*cells, size)
        E = np.exp(rng.uniform(np.log(5e4), np.log(5e5), T.shape[0]))
    s = ps.SimulationSettings()
    s.meshType = "Tetrahedron" if kind == "tet" else "Hexahedron"
    s.dt = 2e-3
    s.timeSteppingScheme = "backward_euler"
    s.solverMethod = method
    s.precision = precision
    s.twoLevelPreconditioner = False
    mask, val = meshes.clamp_mask(X)
    cls = ps.EnergyTet if kind == "tet" else ps.EnergyHex
    en = cls.from_arrays(X, T, s, np.array([0.0, 0.0, -9.81]), 0.0, density=1070.0, youngsModulus=E,
                         poissonsRatio=0.45, neumannBCmask=mask, neumannBCvalue=val)
    v0 = np.where(mask == 1, 0.0, rng.uniform(-0.1, 0.1, X.size))
    en.set_initial_velocity(v0)
    return X, s, en


def _host_newton(en, q, dt):
    import scipy.sparse.linalg as sla
    for _ in range(20):
        g = en.compute_gradient(q, dt)
        H = en.compute_hessian(q, dt)
        d = sla.LinearOperator(H.shape, matvec=lambda v, w=1.0 / H.diagonal(): w * v)
        dx, info = sla.cg(H, -g, rtol=1e-13, atol=0.0, maxiter=20000, M=d)
        assert info == 0
        q = q + dx
        if np.linalg.norm(dx) < 1e-10:
            return q
    raise AssertionError("host Newton did not converge")


@pytest.mark.parametrize("kind,cells,precision", CASES)
def test_step_matches_host_newton(kind, cells, precision):
    from sors_b200 import py_sors as ps
    X, s, en = _energy(kind, cells, precision)
    _, _, ref = _energy(kind, cells, "fp64")
    qr = _host_newton(ref, X.ravel().copy(), s.dt)
    q = ps.Solver(s).step(X.ravel(), en)
    tol = 1e-8 if precision == "fp64" else 1e-6 * np.abs(qr - X.ravel()).max()
    assert np.abs(q - qr).max() <= tol
    # a second handle takes the same step bit for bit
    _, s2, en2 = _energy(kind, cells, precision)
    assert np.array_equal(ps.Solver(s2).step(X.ravel(), en2), q)


@pytest.mark.parametrize("kind,cells,precision", [("tet", (40, 34, 33), "fp64"), ("tet", (57, 43, 41), "mixed"),
                                                  ("hex", (31, 30, 29), "fp64")])
def test_streamed_matrix_matches_minres(kind, cells, precision):
    """Meshes whose matrix streams through shared memory (49k and 107k tet nodes, one and
    two aggregates per range; 30k hex nodes), against MINRES's separate kernels in FP64.
    Both stop at ||dx|| < 1e-9 m; mixed precision is held to 1e-6 of the displacement."""
    from sors_b200 import py_sors as ps
    out = []
    for solver, prec in (("minres", "fp64"), ("pcg", precision), ("pcg", precision)):
        X, s, _ = _energy(kind, (2, 2, 2), prec)
        s.linearSolver = solver
        s.twoLevelPreconditioner = "auto"
        X, en, v0 = _large(kind, cells, s)
        q = ps.Solver(s).step(X.ravel(), en)
        out.append(q)
    tol = 1e-8 if precision == "fp64" else 1e-6 * np.abs(out[0] - X.ravel()).max()
    assert np.abs(out[1] - out[0]).max() <= tol
    assert np.array_equal(out[1], out[2])


def _large(kind, cells, s):
    from sors_b200 import py_sors as ps
    size = tuple(5e-3 * c for c in cells)
    rng = np.random.default_rng(5)
    if kind == "tet":
        X, T, E = meshes.jittered_block_tets(*cells, size, jitter=0.1, seed=5)
    else:
        X, T = meshes.hex_bar(*cells, size)
        E = np.exp(rng.uniform(np.log(5e4), np.log(5e5), T.shape[0]))
    mask, val = meshes.clamp_mask(X)
    cls = ps.EnergyTet if kind == "tet" else ps.EnergyHex
    en = cls.from_arrays(X, T, s, np.array([0.0, 0.0, -9.81]), 0.0, density=1070.0, youngsModulus=E,
                         poissonsRatio=0.45, neumannBCmask=mask, neumannBCvalue=val)
    v0 = np.where(mask == 1, 0.0, rng.uniform(-0.1, 0.1, X.size))
    en.set_initial_velocity(v0)
    return X, en, v0


def test_capped_handle_and_concurrent_streams():
    """Handles whose grids are capped (rollouts side by side) step from four
    threads at once and give the bits they give alone."""
    import threading

    from sors_b200 import py_sors as ps
    out = {}

    def run(k, cells):
        X, s, _ = _energy("tet", cells, "mixed")
        mask, val = meshes.clamp_mask(X)
        s.maxBlocksPerKernel = 148
        en = ps.EnergyTet.from_arrays(X, meshes.kuhn_tet_elements(*cells), s, np.array([0.0, 0.0, -9.81]), 0.0,
                                      density=1070.0, youngsModulus=1e5, poissonsRatio=0.45, neumannBCmask=mask,
                                      neumannBCvalue=val)
        q, sol = X.ravel().copy(), ps.Solver(s)
        for _ in range(3):
            q = sol.step(q, en)
        out[k] = q

    jobs = [(0, (16, 12, 12)), (1, (7, 5, 5)), (2, (18, 16, 16)), (3, (9, 9, 9))]
    for k, c in jobs:
        run(("alone", k), c)
    ts = [threading.Thread(target=run, args=(("mix", k), c)) for k, c in jobs]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for k, _ in jobs:
        assert np.array_equal(out[("alone", k)], out[("mix", k)])


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("mixed", 1e-5)])
def test_hessian_blocks_in_two_pieces(oracle, precision, tol):
    """compute_hessian of a mesh with more blocks than one copy takes (about 250,000,
    against 233,016), in the caller's order, against the oracle.  FP64 to the assembly's
    1e-10; FP32 blocks to 1e-5 of the largest entry (60 items at 6e-8 each, doubled)."""
    from tests.helpers import make_pair
    X = meshes.grid_nodes(25, 25, 25, (0.1, 0.1, 0.1))
    T = meshes.kuhn_tet_elements(25, 25, 25)
    rng = np.random.default_rng(3)
    q = (X @ (np.eye(3) + rng.uniform(-0.05, 0.05, (3, 3))).T).ravel()
    en, _, o, _ = make_pair(X, T, project=False, precision=precision)
    H = en.compute_hessian(q, 1e-3)
    Ho, _ = o.hessian_csr(q, 1e-3)
    d = H - Ho
    assert np.abs(d.data).max() <= tol * np.abs(Ho.data).max()
