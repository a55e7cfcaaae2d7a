"""Timed cases of the implicit-Euler FEM framework, through its public entry points.

Each case is one kind of call that a program makes, with its sizes and options:

  step      Solver.step: a rollout restarted from a state (q, v) and stepped
            `steps` times, Neo-Hookean or stable Neo-Hookean tet blocks clamped
            at x = 0 under gravity (backward Euler or Crank-Nicolson).
  poke      Solver.step with contact (minimize_SQP): the first steps of a poke
            rollout, a cube on the ground plane pressed by a moving disk, as the
            rollout server runs them.
  arm       Solver.step, quasistatic: one load level of a hex arm with three
            pressurised chambers.
  adjoint   RolloutAdjoint.forward and .backward on a muscle-driven hex bar
            that lands on a plane: the gradient with respect to Young's moduli,
            activations and the initial state.
  gradient, energy, hessian
            Energy.compute_gradient / compute_energy / compute_hessian_bsr, for
            programs that bring their own optimiser.
  energy_device
            the element energy of device-resident arrays without allocations
            (sors_elem_energy_noalloc), for real-time loops.

The meshes are the framework's own workload generators (sors_b200.meshes,
sors_b200.serving) with 5 mm cells for the blocks, seeded jitter, material,
velocities and loads.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from sors_b200 import _lib, meshes, serving
from sors_b200 import py_sors as ps
from sors_b200.adjoint import RolloutAdjoint

CELL = 5e-3          # cell size of the tet blocks and hex bars (m)
GRAVITY = (0.0, 0.0, -9.81)
RHO, NU = 1070.0, 0.45
E_RANGE = (5e4, 5e5)
MAX_DENSE_NODES = 4500   # exact() solves steps up to this size with a dense Newton matrix


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the cantilever that every first program steps: 1,920 tets, one step of
        # 1 ms; launches and host round trips count
        dict(name="step cantilever fp64", kind="step", nx=20, ny=4, nz=4, precision="fp64",
             energy="neohookean", scheme="backward_euler", dt=1e-3, steps=1),
        # a calibration-sized block in plain FP64, the drop-in's own precision
        dict(name="step block 21k fp64", kind="step", nx=24, ny=12, nz=12, precision="fp64",
             energy="neohookean", scheme="backward_euler", dt=5e-3, steps=1),
        # the default integrator and the other energy, odd sizes, mixed precision
        dict(name="step snh cn 52k mixed", kind="step", nx=43, ny=15, nz=13, precision="mixed",
             energy="stableneohookean", scheme="crank_nicolson", dt=5e-3, steps=1),
        # a large block with the two-level preconditioner in FP64
        dict(name="step block 120k fp64", kind="step", nx=69, ny=17, nz=17, precision="fp64",
             energy="neohookean", scheme="backward_euler", dt=5e-3, steps=1),
        # the framework's headline workload: the 3.0M-tet block in mixed precision
        dict(name="step block 3.0M mixed", kind="step", nx=200, ny=50, nz=50, precision="mixed",
             energy="neohookean", scheme="backward_euler", dt=5e-3, steps=1),
        # serving: a small and a middle-sized poke cube (8k and 60k tets)
        dict(name="poke 8k mixed", kind="poke", n=11, precision="mixed", steps=4),
        dict(name="poke 59k mixed", kind="poke", n=21, precision="mixed", steps=3),
        # quasistatic actuation of the 200 mm hex arm, 2.5 mm voxels
        dict(name="arm 15k hexes fp64", kind="arm", voxel=2.5e-3, layers=80, precision="fp64"),
        # one gradient of a muscle-driven landing (2,560 hexes)
        dict(name="adjoint bar 2560 hexes", kind="adjoint", nx=40, ny=8, nz=8, steps=3, precision="fp64"),
        # an own optimiser's gradient and Hessian, and a controller's energy
        dict(name="gradient 200k", kind="gradient", nx=81, ny=21, nz=20, precision="fp64"),
        dict(name="hessian 21k", kind="hessian", nx=24, ny=12, nz=12, precision="fp64"),
        dict(name="energy device 60k", kind="energy_device", nx=40, ny=16, nz=16),
    ]


def _block_cells(rng, tets):
    """Cell counts of a beam-like block of about `tets` tets, ragged."""
    a = rng.uniform(1.5, 5.0)
    side = (tets / 6.0 / a) ** (1.0 / 3.0)
    ny = max(2, int(round(side * rng.uniform(0.85, 1.15))))
    nz = max(2, int(round(side * rng.uniform(0.85, 1.15))))
    nx = max(3, int(tets / 6.0 / (ny * nz)))
    return nx, ny, nz


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case of the same ranges: kinds by how often a program makes the
    call (steps most of all), sizes log-uniform."""
    kind = rng.choices(["step", "poke", "arm", "adjoint", "gradient", "energy", "hessian", "energy_device"],
                       [8, 3, 2, 2, 2, 1, 1, 1])[0]
    precision = rng.choice(["fp64", "mixed"])
    if kind == "poke":
        return dict(kind=kind, n=int(round((_log_uniform(rng, 5e3, 2.5e5) / 6.0) ** (1.0 / 3.0))),
                    precision=precision, steps=rng.randint(2, 4))
    if kind == "arm":
        voxel = rng.choice([2.5e-3, 2.5e-3, 1.25e-3])
        return dict(kind=kind, voxel=voxel, layers=rng.randint(16, 80) * int(2.5e-3 / voxel), precision=precision)
    if kind == "adjoint":
        return dict(kind=kind, nx=rng.randint(8, 40), ny=rng.randint(3, 8), nz=rng.randint(3, 8),
                    steps=rng.randint(2, 4), precision="fp64")
    hi = {"step": 2.5e6 if precision == "mixed" else 1e6, "gradient": 1e6, "energy": 1e6, "hessian": 1e5,
          "energy_device": 1e6}[kind]
    nx, ny, nz = _block_cells(rng, _log_uniform(rng, 1.5e3, hi))
    case = dict(kind=kind, nx=nx, ny=ny, nz=nz)
    if kind == "energy_device":
        return case
    case["precision"] = precision
    if kind == "step":
        case.update(energy=rng.choice(["neohookean"] * 3 + ["stableneohookean"]),
                    scheme=rng.choice(["backward_euler"] * 3 + ["crank_nicolson"]),
                    dt=rng.choice([1e-3, 2e-3, 5e-3]), steps=rng.randint(1, 3) if nx * ny * nz < 4000 else 1)
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _block(case, seed):
    size = (case["nx"] * CELL, case["ny"] * CELL, case["nz"] * CELL)
    return meshes.jittered_block_tets(case["nx"], case["ny"], case["nz"], size, jitter=0.1, seed=seed, e_range=E_RANGE)


def _velocity(X, seed):
    """A smooth swing of the beam, zero at its clamped end."""
    rng = np.random.default_rng(seed + 1)
    s = X[:, 0] / X[:, 0].max()
    v = np.zeros_like(X)
    for m in range(2):
        v += rng.uniform(-0.1, 0.1, 3) * np.sin((m + 0.5) * math.pi * s)[:, None]
    return v.ravel()


def _deformed(X, seed):
    """A bent, stretched and slightly rough state of the block (no inverted element)."""
    rng = np.random.default_rng(seed + 2)
    a = rng.uniform(-0.05, 0.05, (3, 3))
    x = X @ (np.eye(3) + a).T
    L = X[:, 0].max()
    x[:, 1:] += rng.uniform(-0.03, 0.03, 2) * L * ((X[:, :1] / L) ** 2)
    return (x + rng.uniform(-0.02, 0.02, X.shape) * CELL).ravel()


def _block_energy(case, seed):
    X, T, E = _block(case, seed)
    s = ps.SimulationSettings()
    s.meshType = "Tetrahedron"
    s.dt = case.get("dt", 5e-3)
    s.timeSteppingScheme = case.get("scheme", "backward_euler")
    s.solverMethod = "minimize_newton"
    s.precision = case["precision"]
    s.newtonResidualTol = 1e-8
    mask, val = meshes.clamp_mask(X)
    en = ps.EnergyTet.from_arrays(X, T, s, np.asarray(GRAVITY), 0.0, density=RHO, youngsModulus=E, poissonsRatio=NU,
                                  neumannBCmask=mask, neumannBCvalue=val, energy=case.get("energy", "neohookean"))
    return X, T, E, en, ps.Solver(s)


def _arm_mesh(case):
    X, H = meshes.voxel_cylinder(radius=0.02, length=case["voxel"] * case["layers"], h=case["voxel"],
                                cap_layers=2)
    groups, _ = meshes.extract_surfaces(X, H)
    groups.pop(int(np.argmax([len(g) for g in groups])))   # the outer skin carries no pressure
    return X, H, groups


def _ptr(a, ct=C.c_double):
    return a.ctypes.data_as(C.POINTER(ct))


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case)
    if kind == "step":
        X, _, _, st["en"], st["sol"] = _block_energy(case, seed)
        st["q0"], st["v0"] = X.ravel().copy(), _velocity(X, seed)
    elif kind in ("gradient", "energy", "hessian"):
        X, _, _, st["en"], _ = _block_energy(case, seed)
        st["en"].set_initial_velocity(_velocity(X, seed))
        st["q"] = _deformed(X, seed)
    elif kind == "energy_device":
        X, T, E = _block(case, seed)
        st["ne"] = T.shape[0]
        st["d"] = [torch.as_tensor(np.ascontiguousarray(a).ravel(), device="cuda")
                   for a in (X, _deformed(X, seed), T, E, np.full(T.shape[0], NU))]
        st["out"] = torch.zeros(1, dtype=torch.float64, device="cuda")
        st["stream"] = torch.cuda.current_stream().cuda_stream
    elif kind == "poke":
        req = serving.poke_cube_request(np.random.default_rng(seed), case["n"], steps=20, precision=case["precision"])
        st["en"], st["sol"], _, st["disks"] = serving.build_union([req])
        st["q0"], st["dt"] = np.ascontiguousarray(req.vertices).ravel(), req.dt
        st["v0"] = np.zeros_like(st["q0"])
        k = _lib.load().sors_get_contact_state(st["en"].handle(), None, 0)
        st["contact0"] = np.zeros(k, np.int32)
        _lib.load().sors_get_contact_state(st["en"].handle(), _ptr(st["contact0"], C.c_int32), k)
    elif kind == "arm":
        rng = np.random.default_rng(seed)
        X, H, groups = _arm_mesh(case)
        s = ps.SimulationSettings()
        s.meshType = "Hexahedron"
        s.dt = 0.0
        s.timeSteppingScheme = "backward_euler"
        s.precision = case["precision"]
        s.hessianProjection = True
        faces = np.concatenate(groups).astype(float)
        gid = np.concatenate([np.full(len(g), float(k)) for k, g in enumerate(groups)])
        fp = ps.Params(["surfaceVertexIdx", "surfaceGroups"], [faces, gid])
        mask = np.repeat((np.abs(X[:, 2]) < 1e-12).astype(np.int32), 3)
        st["en"] = ps.EnergyHex.from_arrays(X, H, s, np.zeros(3), 0.0, density=RHO, youngsModulus=3e5,
                                            poissonsRatio=0.48, neumannBCmask=mask, neumannBCvalue=np.zeros(mask.size),
                                            forceTypesList=["pressure"], forceParameterList=fp)
        st["sol"] = ps.Solver(s)
        st["q0"] = X.ravel().copy()
        pr = np.zeros((len(groups), 1))
        pr[0, 0] = rng.uniform(3e3, 6e3)
        st["act"] = ps.Params(["pressure"], [pr])
    elif kind == "adjoint":
        rng = np.random.default_rng(seed)
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        X, H = meshes.hex_bar(nx, ny, nz, (nx * CELL, ny * CELL, nz * CELL))
        X = X + np.array([0.0, 0.0, 1e-3])
        ne = H.shape[0]
        s = ps.SimulationSettings()
        s.meshType = "Hexahedron"
        s.dt = 2e-3
        s.timeSteppingScheme = "backward_euler"
        s.solverMethod = "minimize_SQP"
        s.precision = case["precision"]
        st["en"] = ps.EnergyHex.from_arrays(X, H, s, np.asarray(GRAVITY), 0.0, density=RHO, youngsModulus=2e5,
                                            poissonsRatio=NU, muscleGroup=np.arange(ne),
                                            softconStiffness=np.full(ne, 5e4),
                                            softconDirection=np.tile([1.0, 0.0, 0.0], (ne, 1)))
        surf, _ = meshes.extract_surfaces(X, H)
        cp = ps.Params(["positionVectorListPlanes", "normalVectorListPlanes", "surfaceVerticesIdx"],
                       [np.zeros(3), np.array([0.0, 0.0, 1.0]), np.unique(np.concatenate(surf)).astype(float)])
        st["en"]._setup_constraints_forces(["planeContact"], cp, (), None)
        v0 = np.tile([0.0, 0.0, -0.5], X.shape[0]) + rng.uniform(-0.01, 0.01, X.size)
        st["roll"] = RolloutAdjoint(st["en"], ps.Solver(s), case["steps"], 2e-3, v0=v0, poisson=NU, checkpoint_every=2)
        st["E"] = 2e5 * rng.uniform(0.8, 1.25, ne)
        st["act"] = rng.uniform(0.0, 1.0, (case["steps"], ne))
        st["dL"] = rng.standard_normal(X.size) / X.shape[0]
    else:
        raise ValueError(kind)
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _restart(st):
    st["en"].set_initial_deformation(st["q0"])
    st["en"].set_initial_velocity(st["v0"])


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "step":
        _restart(st)
        if case["scheme"] == "crank_nicolson":
            z = np.zeros_like(st["q0"])
            _lib.check(_lib.load().sors_set_prev_force(st["en"].handle(), _ptr(z)))
        q = st["q0"]
        for _ in range(case["steps"]):
            q = st["sol"].step(q, st["en"])
        return q
    if kind == "gradient":
        return st["en"].compute_gradient(st["q"], 5e-3)
    if kind == "energy":
        return np.array([st["en"].compute_energy(st["q"], 5e-3)])
    if kind == "hessian":
        rp, col, blocks = st["en"].compute_hessian_bsr(st["q"], 5e-3)
        return dict(row_ptr=rp, col=col, blocks=blocks)
    if kind == "energy_device":
        X, q, T, E, nu = (C.c_void_p(t.data_ptr()) for t in st["d"])
        _lib.check(_lib.load().sors_elem_energy_noalloc(X, q, T, st["ne"], 4, E, nu, C.c_void_p(st["out"].data_ptr()),
                                                        C.c_void_p(st["stream"])))
        return st["out"]
    if kind == "poke":
        _restart(st)
        c = st["contact0"]
        _lib.check(_lib.load().sors_set_contact_state(st["en"].handle(), _ptr(c, C.c_int32), c.size))
        q = st["q0"]
        for t in range(case["steps"]):
            for d, (c0, nrm, rad, vel) in enumerate(st["disks"]):
                serving._lib_set_disk(st["en"], d, c0 + vel * st["dt"] * t, nrm, rad)
            q = st["sol"].step(q, st["en"])
        return q
    if kind == "arm":
        return st["sol"].step(st["q0"], st["en"], st["act"], 0.0)
    if kind == "adjoint":
        qT = st["roll"].forward(st["E"], st["act"])
        gE, gA, gq, gv = st["roll"].backward(st["dL"])
        return dict(q=qT, gE=gE, gA=gA, gq=gq, gv=gv)
    raise ValueError(kind)


# ---------------------------------------------------------------------------
# what one pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: positions, velocities, connectivity and material in, the result
    out, once per step (and the Hessian where it is the result); operations:
    one evaluation of every element (a tet's gradient about 250 operations and
    its Hessian 600 more, eight points of a hex) and one block matrix-vector
    product per implicit step."""
    kind = case["kind"]
    if kind == "arm":
        k = (2.5e-3 / case["voxel"]) ** 2
        ne = 180 * k * case["layers"]
        nodes = 220 * k * (case["layers"] + 1)
        return dict(bytes=48.0 * ne + 72.0 * nodes, flops=8.0 * 3000 * ne + 18.0 * 24 * nodes)
    if kind == "poke":
        case = dict(case, nx=case["n"], ny=case["n"], nz=case["n"])
    cells = case["nx"] * case["ny"] * case["nz"]
    nodes = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
    if kind == "adjoint":
        per = 72.0 * cells + 120.0 * nodes
        return dict(bytes=2 * case["steps"] * per, flops=2.0 * case["steps"] * (8 * 3000 * cells + 18 * 24 * nodes))
    ne, nnzb = 6 * cells, 15 * nodes
    steps = case.get("steps", 1)
    if kind in ("step", "poke"):
        return dict(bytes=steps * (32.0 * ne + 96.0 * nodes), flops=steps * (850.0 * ne + 18.0 * nnzb))
    if kind == "energy_device":
        return dict(bytes=32.0 * ne + 48.0 * nodes + 8, flops=150.0 * ne)
    if kind == "energy":
        return dict(bytes=32.0 * ne + 104.0 * nodes, flops=150.0 * ne + 30.0 * nodes)
    if kind == "gradient":
        return dict(bytes=32.0 * ne + 128.0 * nodes, flops=250.0 * ne + 30.0 * nodes)
    return dict(bytes=32.0 * ne + 128.0 * nodes + 76.0 * nnzb, flops=850.0 * ne)


# ---------------------------------------------------------------------------
# 64-bit values without the framework's kernels
# ---------------------------------------------------------------------------
class _TetSystem:
    """Neo-Hookean tets in plain torch: lumped mass, backward Euler, clamped nodes."""

    def __init__(self, X, T, E, dt, dev="cuda"):
        self.X = torch.as_tensor(X, device=dev)
        self.T = torch.as_tensor(T.astype(np.int64), device=dev)
        self.n = X.shape[0]
        Dm = (self.X[self.T[:, :3]] - self.X[self.T[:, 3:]]).transpose(1, 2)
        self.V = torch.linalg.det(Dm).abs() / 6.0
        B = torch.linalg.inv(Dm)
        self.D = torch.cat([B, -B.sum(1, keepdim=True)], 1)      # shape gradients, (E, 4, 3)
        E = torch.as_tensor(E, device=dev)
        self.mu, self.lam = E / (2 * (1 + NU)), E * NU / ((1 + NU) * (1 - 2 * NU))
        self.m = torch.zeros(self.n, dtype=torch.float64, device=dev)
        self.m.index_add_(0, self.T.ravel(), (RHO * self.V / 4.0).repeat_interleave(4))
        self.g = torch.tensor(GRAVITY, dtype=torch.float64, device=dev)
        self.dt = dt
        self.fixed = (self.X[:, 0] - self.X[:, 0].min()).abs() <= 1e-9

    def F(self, x):
        return torch.einsum("ewr,ewc->erc", x[self.T], self.D)

    def element_energy(self, x):
        F = self.F(x)
        lj = torch.log(torch.linalg.det(F))
        return (self.V * (0.5 * self.mu * ((F * F).sum((1, 2)) - 3.0) - self.mu * lj + 0.5 * self.lam * lj * lj)).sum()

    def elastic_gradient(self, x):
        F = self.F(x)
        lj = torch.log(torch.linalg.det(F))
        P = self.mu[:, None, None] * F + (self.lam * lj - self.mu)[:, None, None] * torch.linalg.inv(F).transpose(1, 2)
        f = torch.einsum("e,erc,ewc->ewr", self.V, P, self.D)
        out = torch.zeros_like(x)
        out.index_add_(0, self.T.ravel(), f.reshape(-1, 3))
        return out

    def element_hessians(self, x):
        """(E, 4, 3, 4, 3)"""
        F = self.F(x)
        lj = torch.log(torch.linalg.det(F))
        a = torch.einsum("ecr,ewc->ewr", torch.linalg.inv(F), self.D)      # F^-T d_w
        eye = torch.eye(3, dtype=torch.float64, device=x.device)
        dd = torch.einsum("evc,ewc->evw", self.D, self.D)
        K = torch.einsum("e,evw,kl->evkwl", self.mu, dd, eye)
        K += torch.einsum("e,evk,ewl->evkwl", self.lam, a, a)
        K -= torch.einsum("e,ewk,evl->evkwl", self.lam * lj - self.mu, a, a)
        return K * self.V[:, None, None, None, None]

    def gradient(self, x, xp, vp):
        v = (x - xp) / self.dt
        g = self.elastic_gradient(x) + self.m[:, None] * ((v - vp) / self.dt - self.g)
        return torch.where(self.fixed[:, None], x - xp, g)

    def energy(self, x, xp, vp):
        acc = ((x - xp) / self.dt - vp) / self.dt
        return (self.element_energy(x) - (self.m[:, None] * x * self.g).sum()
                + 0.5 * self.dt ** 2 * (self.m[:, None] * acc * acc).sum())

    def step(self, xp, vp):
        n3 = 3 * self.n
        x = xp.clone()
        dof = (3 * self.T[:, :, None] + torch.arange(3, device=x.device)).reshape(-1, 12)
        at = (dof[:, :, None] * n3 + dof[:, None, :]).ravel()
        free = torch.nonzero(~self.fixed.repeat_interleave(3)).ravel()
        inertia = self.m.repeat_interleave(3) / self.dt ** 2
        for _ in range(40):
            H = torch.zeros(n3 * n3, dtype=torch.float64, device=x.device)
            H.index_add_(0, at, self.element_hessians(x).reshape(-1))
            H = H.reshape(n3, n3)
            H.diagonal().add_(inertia)
            dx = torch.zeros(n3, dtype=torch.float64, device=x.device)
            dx[free] = torch.linalg.solve(H[free][:, free], -self.gradient(x, xp, vp).ravel()[free])
            x = x + dx.reshape(-1, 3)
            if float(dx.norm()) < 1e-12:
                break
        return x, (x - xp) / self.dt


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("step", "gradient", "energy", "hessian", "energy_device"):
        return None
    if case.get("energy", "neohookean") != "neohookean" or case.get("scheme", "backward_euler") != "backward_euler":
        return None
    nodes = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
    if kind == "step" and nodes > MAX_DENSE_NODES:
        return None
    X, T, E = _block(case, seed)
    s = _TetSystem(X, T, E, case.get("dt", 5e-3))
    v = torch.as_tensor(_velocity(X, seed), device="cuda").reshape(-1, 3)
    if kind == "step":
        x = s.X
        for _ in range(case["steps"]):
            x, v = s.step(x, v)
        return x.ravel().cpu().numpy()
    q = torch.as_tensor(_deformed(X, seed), device="cuda").reshape(-1, 3)
    if kind == "gradient":
        return s.gradient(q, s.X, v).ravel().cpu().numpy()
    if kind == "energy":
        return np.array([float(s.energy(q, s.X, v))])
    if kind == "energy_device":
        return s.element_energy(q).reshape(1)
    # the 3x3 blocks in CSR order: columns ascending in each row; clamped rows and columns are the identity's
    n = s.n
    rows = s.T[:, :, None].expand(-1, 4, 4).reshape(-1)
    cols = s.T[:, None, :].expand(-1, 4, 4).reshape(-1)
    key, inv = torch.unique(rows * n + cols, return_inverse=True)
    blocks = torch.zeros(key.numel(), 3, 3, dtype=torch.float64, device="cuda")
    blocks.index_add_(0, inv, s.element_hessians(q).permute(0, 1, 3, 2, 4).reshape(-1, 3, 3))
    i, j = key // n, key % n
    blocks[s.fixed[i] | s.fixed[j]] = 0.0
    eye = torch.eye(3, dtype=torch.float64, device="cuda")
    d = i == j
    blocks[d] += torch.where(s.fixed, 1.0, s.m / s.dt ** 2)[i[d]][:, None, None] * eye
    return dict(row_ptr=None, col=None, blocks=blocks.cpu().numpy())
