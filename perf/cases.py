"""Performance cases of the solve path, through the package's public entry points.

Each case is one call, or one step of a loop, that a program built on the
framework makes: a job that is read, solved and closed, a design iteration
(new moduli, assembly, solve, gradient), a transient run with and without its
reverse sweep, a frequency job, a batched sweep, a training step.  Kinds:

  job        one small beam, the job runner's defaults (FP64 point-Jacobi CG to
             1e-12), tip objective, per-element and grouped modulus gradients
  oneshot    a whole job on a tetrahedral mesh: context, pattern, assembly,
             solve, element stresses, close (nothing is kept between jobs)
  multicase  several load cases on one hex8 model, the Python default method
             (mixed precision, point Jacobi)
  design     a design / UQ step on a hex8 block: FP64-accurate split operator,
             multigrid CG, compliance and its modulus gradient
  brickim    the same with the reference's default hex (incompatible modes) and
             a tip-displacement objective (a second, adjoint solve)
  learned    a held-out field of the learned-preconditioner grid: multigrid CG
             with network-predicted finest smoother blocks
  batch      uneven cantilevers stacked in one operator, four load cases each
  newmark    a shell plate under a central impulse (transient, FP64)
  transient  a hex8 beam's Newmark run with its history kept, and the reverse
             (adjoint) sweep over it
  modal      the lowest eigenvalues of a hex8 block (shift-invert Lanczos on
             multigrid CG)
  train      residual samples and the loss gradient of the learned smoother on
             a training patch

The moduli of a case are a seeded lognormal field; a pass hands them over from
host memory and returns host arrays, as the C ABI does.  The solver handle
(mesh, pattern, hierarchy) is what such a program keeps, except in `oneshot`.
"""
import math

import numpy as np
import torch

from asend3d_gb300 import _lib, configs, learned
from asend3d_gb300.mesh import block_hex8, block_tet4, lognormal_modulus
from asend3d_gb300.solver import GpuSolver, Problem, combine

# Newmark parameters of the benchmark's plate and of the transient beam
# (beta in the reference's convention), and the beam's time step
PLATE_DT, BEAM_DT, BETA, GAMMA = 2e-6, 2e-4, 0.25, 0.5

SPLIT_MG = dict(method=_lib.METHOD_SPLIT, precond=_lib.PC_MG, rel_tol=3e-10, graph_iters=8)
JACOBI64 = dict(method=_lib.METHOD_FP64, precond=_lib.PC_JACOBI)


def listed():
    return [
        # the smallest call: a 320-element beam, latency and launches
        dict(name="job_beam_20x4x4", kind="job", nx=20, ny=4, nz=4),
        # an ordinary single job on an unstructured (tetrahedral) mesh, nothing kept
        dict(name="oneshot_tet_30x7x6", kind="oneshot", nx=30, ny=7, nz=6),
        # six load cases at once (a chunk of four and a remainder of two)
        dict(name="multicase_61x9x7", kind="multicase", nx=61, ny=9, nz=7, cases=6),
        # an ordinary design step, and the benchmark's million-DOF block
        dict(name="design_100x20x20", kind="design", nx=100, ny=20, nz=20),
        dict(name="design_200x40x40", kind="design", nx=200, ny=40, nz=40),
        # the reference's default hex, odd sizes
        dict(name="brickim_57x13x11", kind="brickim", nx=57, ny=13, nz=11),
        # the largest: 1.6 million DOF, rougher field
        dict(name="learned_128x64x64", kind="learned", nx=128, ny=64, nz=64),
        # an uneven stack (a quarter of the 64-instance sweep)
        dict(name="batch_16x4", kind="batch", instances=16),
        # transient plate: 61,206 DOF, launch-bound steps
        dict(name="newmark_plate_100", kind="newmark", n=100, steps=60),
        # forward and reverse sweep of a beam
        dict(name="transient_beam_24x6x6", kind="transient", nx=24, ny=6, nz=6, steps=40),
        # a frequency job
        dict(name="modal_60x12x9", kind="modal", nx=60, ny=12, nz=9, modes=6),
        # one training field of the learned smoother
        dict(name="train_patch_16x8x8", kind="train", nx=16, ny=8, nz=8),
    ]


def draw(rng):
    def size(lo, hi):  # log-uniform whole number in [lo, hi]
        return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    kind = rng.choice(["job", "oneshot", "multicase", "design", "design", "brickim", "learned", "batch", "newmark",
                       "transient", "modal", "train"])
    if kind == "job":
        return dict(kind=kind, nx=size(8, 40), ny=size(2, 6), nz=size(2, 6))
    if kind == "oneshot":
        return dict(kind=kind, nx=size(12, 48), ny=size(3, 9), nz=size(3, 9))
    if kind == "multicase":
        return dict(kind=kind, nx=size(20, 80), ny=size(4, 10), nz=size(4, 10), cases=rng.randint(2, 7))
    if kind == "design":
        return dict(kind=kind, nx=size(40, 200), ny=size(8, 40), nz=size(8, 40))
    if kind == "brickim":
        return dict(kind=kind, nx=size(24, 96), ny=size(6, 18), nz=size(6, 18))
    if kind == "learned":
        n = size(24, 64)
        return dict(kind=kind, nx=size(48, 128), ny=n, nz=n)
    if kind == "batch":
        return dict(kind=kind, instances=size(4, 16))
    if kind == "newmark":
        return dict(kind=kind, n=size(24, 140), steps=rng.randint(20, 60))
    if kind == "transient":
        return dict(kind=kind, nx=size(10, 32), ny=size(2, 7), nz=size(2, 7), steps=rng.randint(20, 40))
    if kind == "modal":
        return dict(kind=kind, nx=size(24, 72), ny=size(8, 12), nz=size(5, 7), modes=rng.randint(4, 8))
    return dict(kind=kind, nx=size(12, 32), ny=size(6, 12), nz=size(6, 12))


# ---------------------------------------------------------------------------
# the models
# ---------------------------------------------------------------------------
def _tet_problem(case, seed):
    """A fixed-end tetrahedral bar with a transverse force spread over its end."""
    m = block_tet4(case["nx"], case["ny"], case["nz"], *configs.BAR)
    p = Problem(m, lognormal_modulus(m, 70e9, 0.3, 0.1, seed), np.full(m.n_elems, 0.33),
                np.full(m.n_elems, 2700.0))
    configs._fixed_end(p, m)
    end = m.nodes_in_range(xr=(configs.BAR[0] - 1e-9, configs.BAR[0] + 1e-9))
    p.add_node_set("xMax", end)
    p.add_nodal_force("xMax", [0.0, 0.0, -1000.0 / len(end)])
    return p


def _problem(case, seed):
    kind = case["kind"]
    if kind == "job":
        p = configs.cantilever_small(case["nx"], case["ny"], case["nz"])
        p.E = lognormal_modulus(p.mesh, 200e9, 0.2, 0.2, seed)
        return p
    if kind == "oneshot":
        return _tet_problem(case, seed)
    if kind == "multicase":
        p = configs.block_large(case["nx"], case["ny"], case["nz"], seed=seed)
        m = p.mesh
        end = m.nodes_in_range(xr=(configs.BAR[0] - 1e-9, configs.BAR[0] + 1e-9))
        p.add_node_set("xMax", end)
        rng = np.random.default_rng([seed, 1])
        p.loads = []
        for k in range(case["cases"]):  # end forces in seeded directions
            p.add_nodal_force("xMax", 1000.0 * rng.standard_normal(3) / len(end), case=k)
        return p
    if kind in ("design", "modal"):
        return configs.block_large(case["nx"], case["ny"], case["nz"], seed=seed)
    if kind == "brickim":
        p = configs.block_large(case["nx"], case["ny"], case["nz"], seed=seed)
        p.mesh.elem_type = 81
        tip = p.mesh.nodes_in_range(xr=(configs.BAR[0] - 1e-9, configs.BAR[0] + 1e-9))
        p.add_node_set("tip", tip)
        p.objective = ("displacement", "tip", 3, 1.0 / len(tip))
        return p
    if kind in ("learned", "train"):
        return configs.learned_patch(case["nx"], case["ny"], case["nz"], seed=seed)
    if kind == "newmark":
        p = configs.shell_plate(case["n"])
        rng = np.random.default_rng([seed, 2])
        p.E = p.E * np.exp(0.1 * rng.standard_normal(p.mesh.n_elems))
        return p
    if kind == "transient":
        m = block_hex8(case["nx"], case["ny"], case["nz"], 1.0, 0.25, 0.25)
        p = Problem(m, lognormal_modulus(m, 70e9, 0.2, 0.2, seed), np.full(m.n_elems, 0.3), np.full(m.n_elems, 2700.0))
        configs._fixed_end(p, m)
        tip = m.nodes_in_range(xr=(1.0 - 1e-9, 1.0 + 1e-9))
        p.add_node_set("tip", tip)
        p.add_nodal_force("tip", [0.0, 0.0, -1000.0 / len(tip)])
        return p
    raise ValueError(kind)


def _batch_instances(case, seed):
    """Instances of the sweep with their own fields; the shapes do not depend on the seed."""
    out = [configs.batch_instance(k) for k in range(case["instances"])]
    for k, p in enumerate(out):
        p.E = lognormal_modulus(p.mesh, 70e9, 0.3, 0.1, 1000 * seed + k)
    return out


def _transient_load(case):
    return np.sin(np.linspace(0.0, 3.0, case["steps"]))


def _plate_load(case):
    """The part of the benchmark's pulse that carries it, over the case's steps."""
    return configs.gaussian_pulse(case["steps"], PLATE_DT, width=15e-6, t0=50e-6)


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": dict(case), "seed": int(seed)}
    if kind == "oneshot":
        s["problem"] = _tet_problem(case, seed)
        return s
    if kind == "batch":
        inst = _batch_instances(case, seed)
        prob, node_ptr, elem_ptr = combine(inst)
        s["solver"] = g = GpuSolver(prob, instances=node_ptr, blocks=[(p.mesh.nx, p.mesh.ny, p.mesh.nz) for p in inst])
        s["E"] = prob.E
    else:
        p = _problem(case, seed)
        s["solver"] = g = GpuSolver(p)
        s["E"] = p.E
    if kind == "newmark":
        g.assemble(dynamic=True, dt=PLATE_DT, beta=BETA, gamma=GAMMA)
        s["amp"] = _plate_load(case)
        s["probe"] = 6 * int(g.p.node_sets["centre"][0]) + 2
    elif kind == "transient":
        g.assemble(dynamic=True, dt=BEAM_DT, beta=BETA, gamma=GAMMA)
        g.keep_history(1)
        s["amp"] = _transient_load(case)
        s["dofs"] = 3 * g.p.node_sets["tip"] + 2
    elif kind == "modal":
        g.assemble(precision=64, dynamic=2)
    else:
        if kind in ("learned", "train"):
            g.set_learned_params(learned.initial_weights(g, 0))
            g.learned_set_objective(_lib.LEARN_MG)
        g.assemble(precision=64 if kind in ("job", "multicase", "train") else 48)
    return s


def _gradient_step(g, E, precision, **opts):
    g.set_modulus(E)
    g.assemble(precision=precision)
    u, _, _ = g.static_solve(**opts)
    L, dLdE, _, _ = g.adjoint_gradient(**opts)
    return {"u": u, "L": np.array([L]), "dLdE": dLdE}


def run(state):
    kind = state["kind"]
    if kind == "oneshot":
        g = GpuSolver(state["problem"])
        g.assemble(precision=64)
        u, _, _ = g.static_solve(rel_tol=1e-10, **JACOBI64)
        eps, sig, vol = g.element_fields()
        g.close()
        return {"u": u, "strain": eps, "stress": sig, "volume": vol}
    g = state["solver"]
    if kind == "job":
        out = _gradient_step(g, state["E"], 64, rel_tol=1e-12, **JACOBI64)
        out["dLdD"] = g.design_var_gradient(out["dLdE"])
        return out
    if kind == "multicase":
        g.set_modulus(state["E"])
        g.assemble()
        u, _, _ = g.static_solve(rel_tol=1e-10)
        return {"u": u}
    if kind in ("design", "brickim", "batch"):
        return _gradient_step(g, state["E"], 48, **SPLIT_MG)
    if kind == "learned":
        return _gradient_step(g, state["E"], 48, **dict(SPLIT_MG, precond=_lib.PC_MG_LEARNED))
    if kind == "newmark":
        hist, u, _, _ = g.newmark(state["amp"], probe_dof=state["probe"], rel_tol=1e-11, warm_start=2, **JACOBI64)
        return {"history": hist, "u": u}
    if kind == "transient":
        w = np.full(len(state["dofs"]), 1.0 / len(state["dofs"]))
        hist, u, _, _ = g.newmark(state["amp"], probe_dof=int(state["dofs"][0]), rel_tol=1e-12, **JACOBI64)
        L, dLdE, _, _ = g.newmark_adjoint(state["dofs"], w, rel_tol=1e-12, **JACOBI64)
        return {"history": hist, "u": u, "L": np.array([L]), "dLdE": dLdE}
    if kind == "modal":
        g.set_modulus(state["E"])
        g.assemble(precision=64, dynamic=2)
        ev, fr, _, dm, _, _ = g.eigen(state["case"]["modes"], modes=False, tol=1e-8, method=_lib.METHOD_FP64,
                                      precond=_lib.PC_MG, rel_tol=1e-10, max_iter=300)
        return {"eigenvalues": ev, "frequencies": fr, "mass": dm}
    g.set_modulus(state["E"])
    g.assemble(precision=64)
    g.learned_add_samples((0, 0, -4, -8), seed=state["seed"])
    loss, grad = g.learned_loss_grad()
    return {"loss": np.array([loss], dtype=np.float32), "grad": grad}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: the case's inputs (moduli, loads) read once, its operator written
    and read once in FP64 (or FP32 pairs) with its column indices, and its
    results written once; a transient reads the operator once a step.  Flops:
    the operator's products that no exact method avoids: one per solve."""
    kind = case["kind"]
    if kind == "batch":
        sizes = [configs.batch_dims(k) for k in range(case["instances"])]
        cells = sum(a * b * c for a, b, c in sizes)
        nodes = sum((a + 1) * (b + 1) * (c + 1) for a, b, c in sizes)
        entries = sum((3 * a + 1) * (3 * b + 1) * (3 * c + 1) for a, b, c in sizes)
    elif kind == "newmark":
        n = case["n"]
        cells, nodes, entries = n * n, 2 * (n + 1) ** 2, 4 * (3 * n + 1) ** 2
    else:
        a, b, c = case["nx"], case["ny"], case["nz"]
        cells, nodes = a * b * c, (a + 1) * (b + 1) * (c + 1)
        entries = (3 * a + 1) * (3 * b + 1) * (3 * c + 1)
        if kind == "oneshot":  # 6 tetrahedra a cell; 7 edges a node and itself
            cells, entries = 6 * cells, 15 * nodes
    dof, matrix = 3 * nodes, entries * (9 * 8 + 4)
    solves, steps = 1, 1
    if kind in ("job", "brickim"):
        solves = 2
    elif kind == "multicase":
        solves = case["cases"]
    elif kind == "batch":
        solves = 4
    elif kind == "modal":
        solves = case["modes"]
    elif kind == "train":
        solves = 4
    elif kind == "newmark":
        solves = steps = case["steps"]
    elif kind == "transient":
        solves, steps = 2 * case["steps"], 2 * case["steps"]
    out = 8 * cells + 8 * dof * (solves if kind in ("multicase", "batch") else 1)
    if kind == "oneshot":
        out += 8 * 13 * cells
    return {"bytes": 8.0 * cells + 8.0 * dof + matrix * (1.0 + steps) + out, "flops": 18.0 * entries * solves}


# ---------------------------------------------------------------------------
# the same results in 64 bits, from the element formulas and a direct solver
# ---------------------------------------------------------------------------
_CORNER = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1],
                    [-1, 1, 1]], dtype=np.float64)
_GP = 1.0 / math.sqrt(3.0)


def _solid_c(nu):
    """Isotropic stiffness at unit modulus, Voigt 11,22,33,12,13,23."""
    lam, mu = nu / ((1 + nu) * (1 - 2 * nu)), 1 / (2 * (1 + nu))
    C = np.diag([2 * mu] * 3 + [mu] * 3)
    C[:3, :3] += lam
    return C


def _solid_b(g):
    """6 x 3n strain matrix of the n functions with gradients g [n, 3]."""
    B = np.zeros((6, 3 * len(g)))
    x, y, z = g[:, 0], g[:, 1], g[:, 2]
    B[0, 0::3], B[1, 1::3], B[2, 2::3] = x, y, z
    B[3, 0::3], B[3, 1::3] = y, x
    B[4, 0::3], B[4, 2::3] = z, x
    B[5, 1::3], B[5, 2::3] = z, y
    return B


def _hex_matrices(h, nu, incompatible=False):
    """Stiffness at unit modulus and mass at unit density of a box element
    with edges h (nine condensed modes 1 - s_k^2 if incompatible)."""
    h = np.asarray(h, dtype=np.float64)
    C, det = _solid_c(nu), float(np.prod(h)) / 8
    nd = 33 if incompatible else 24
    K, M = np.zeros((nd, nd)), np.zeros((24, 24))
    for s in _CORNER * _GP:
        f = 1 + _CORNER * s
        N = f.prod(axis=1) / 8
        d = np.stack([_CORNER[:, 0] * f[:, 1] * f[:, 2], _CORNER[:, 1] * f[:, 0] * f[:, 2],
                      _CORNER[:, 2] * f[:, 0] * f[:, 1]], axis=1) / 8 * (2 / h)
        if incompatible:
            d = np.concatenate([d, np.diag(-2 * s * (2 / h))])
        B = _solid_b(d)
        K += B.T @ C @ B * det
        M += np.kron(np.outer(N, N), np.eye(3)) * det
    if incompatible:
        K = K[:24, :24] - K[:24, 24:] @ np.linalg.solve(K[24:, 24:], K[24:, :24])
    return K, M


def _shell_matrices(hx, hy, nu, t):
    """Plate element (u v w and three rotations a node, eight condensed modes)
    at unit modulus, and its mass at unit density."""
    G, q, D = 1 / (2 * (1 + nu)), 1 / (1 - nu * nu), t ** 3 / 12
    Q = np.array([[q, nu * q, 0], [nu * q, q, 0], [0, 0, G]])
    C = np.zeros((9, 9))
    C[:3, :3], C[3:6, 3:6] = t * Q, D * Q
    C[6, 6] = C[7, 7] = C[8, 8] = t * G
    det = hx * hy / 4
    K, M = np.zeros((32, 32)), np.zeros((24, 24))
    for s, r in ((-_GP, -_GP), (_GP, -_GP), (-_GP, _GP), (_GP, _GP)):
        N = np.array([(1 - s) * (1 - r), (1 + s) * (1 - r), (1 + s) * (1 + r), (1 - s) * (1 + r)]) / 4
        ds = np.array([-(1 - r) / 4, (1 - r) / 4, (1 + r) / 4, -(1 + r) / 4, -2 * s, 0, -2 * s * (1 - r), 1 - r * r,
                       -2 * s * (1 + r), -1 + r * r])
        dr = np.array([-(1 - s) / 4, -(1 + s) / 4, (1 + s) / 4, (1 - s) / 4, 0, -2 * r, -1 + s * s, -2 * r * (1 + s),
                       1 - s * s, -2 * r * (1 - s)])
        dx, dy = ds * 2 / hx, dr * 2 / hy
        B = np.zeros((9, 32))
        modes = [(4, 0), (5, 0), (4, 1), (5, 1), (6, 2), (7, 2), (8, 2), (9, 2)]
        for col, f, c in [(6 * a + c, a, c) for a in range(4) for c in range(6)] + [
                (24 + k, f, c) for k, (f, c) in enumerate(modes)]:
            x, y = dx[f], dy[f]
            if c == 0:
                B[[0, 2, 8], col] = x, y, y
            elif c == 1:
                B[[1, 2, 8], col] = y, x, -x
            elif c == 2:
                B[[6, 7], col] = x, y
            elif c == 3:
                B[[4, 5, 7], col] = -y, -x, -N[f]
            elif c == 4:
                B[[3, 5, 6], col] = x, y, N[f]
            else:
                B[8, col] = 2 * N[f]
        K += B.T @ C @ B * det
        M += np.kron(np.outer(N, N), np.diag([t] * 3 + [D] * 3)) * det
    return K[:24, :24] - K[:24, 24:] @ np.linalg.solve(K[24:, 24:], K[24:, :24]), M


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _Planes:
    """Symmetric matrix of a mesh numbered plane by plane along x: blocks D of
    the planes and U from each plane to the next; block Cholesky."""

    def __init__(self, conn, plane_nodes, dpn, scale, mats, which=None):
        conn = torch.as_tensor(np.asarray(conn, dtype=np.int64), device=_device())
        self.m, self.P = plane_nodes * dpn, int(conn.max()) // plane_nodes + 1
        m = self.m
        dof = (conn[:, :, None] * dpn + torch.arange(dpn, device=conn.device)).reshape(len(conn), -1)
        mats = torch.as_tensor(np.atleast_3d(mats) if np.ndim(mats) == 3 else np.asarray(mats)[None], device=conn.device)
        scale = torch.as_tensor(np.asarray(scale, dtype=np.float64), device=conn.device)
        which = torch.zeros(len(conn), dtype=torch.long) if which is None else torch.as_tensor(which, dtype=torch.long)
        which = which.to(conn.device)
        self.dof, self.mats, self.which = dof, mats, which
        self.D = torch.zeros(self.P * m * m, dtype=torch.float64, device=conn.device)
        self.U = torch.zeros(max(1, self.P - 1) * m * m, dtype=torch.float64, device=conn.device)
        for e0 in range(0, len(conn), 20000):
            d = dof[e0:e0 + 20000]
            v = scale[e0:e0 + 20000, None, None] * mats[which[e0:e0 + 20000]]
            r, c = torch.broadcast_tensors(d[:, :, None], d[:, None, :])
            pr, pc = r // m, c // m
            at = (pr * m + r % m) * m + c % m
            for out, keep in ((self.D, pr == pc), (self.U, pc == pr + 1)):
                out.index_add_(0, at[keep], v[keep])
        self.D, self.U = self.D.view(self.P, m, m), self.U.view(-1, m, m)

    def largest(self):
        return max(float(self.D.abs().max()), float(self.U.abs().max()) if self.P > 1 else 0.0)

    def add_diagonal(self, dofs, value):
        dofs = torch.as_tensor(np.asarray(dofs, dtype=np.int64), device=self.D.device)
        self.D[dofs // self.m, dofs % self.m, dofs % self.m] += value

    def factor(self):
        self.L, self.W = [], []
        for p in range(self.P):
            S = self.D[p]
            if p:
                self.W.append(torch.linalg.solve_triangular(self.L[-1], self.U[p - 1], upper=False))
                S = S - self.W[-1].T @ self.W[-1]
            self.L.append(torch.linalg.cholesky(S))
        return self

    def _sweep(self, b):
        y = list(b.view(self.P, self.m, -1))
        for p in range(self.P):
            if p:
                y[p] = y[p] - self.W[p - 1].T @ y[p - 1]
            y[p] = torch.linalg.solve_triangular(self.L[p], y[p], upper=False)
        for p in reversed(range(self.P)):
            if p + 1 < self.P:
                y[p] = y[p] - self.W[p] @ y[p + 1]
            y[p] = torch.linalg.solve_triangular(self.L[p].T, y[p], upper=True)
        return torch.stack(y).view(self.P * self.m, -1)

    def times(self, x):
        x = x.view(self.P, self.m, -1)
        y = self.D @ x
        if self.P > 1:
            y[:-1] += self.U @ x[1:]
            y[1:] += self.U.transpose(1, 2) @ x[:-1]
        return y.reshape(self.P * self.m, -1)

    def solve(self, b, refine=1):
        x = self._sweep(b)
        for _ in range(refine):
            x = x + self._sweep(b - self.times(x))
        return x

    def energy(self, a, b):
        """a_e^T K^ b_e per element at unit scale, summed over columns."""
        out = torch.zeros(len(self.dof), dtype=torch.float64, device=self.D.device)
        for k in range(len(self.mats)):
            sel = self.which == k
            ae, be = a[self.dof[sel]], b[self.dof[sel]]
            out[sel] = torch.einsum("eic,ij,ejc->e", ae, self.mats[k], be)
        return out


def _host(x):
    return x.cpu().numpy()


def _loads(p):
    """Load vectors [n_dof, cases] of the problem (nodal forces, end tractions, raw vectors)."""
    m, dpn = p.mesh, p.mesh.dpn
    F = np.zeros((m.n_dof, len(p.loads)))
    for k, items in enumerate(p.loads):
        for it in items:
            if it[0] == "nodalForce":
                for c in range(dpn):
                    np.add.at(F[:, k], dpn * p.node_sets[it[1]] + c, it[2][c])
            elif it[0] == "vector":
                F[:, k] += it[1]
            else:  # traction on the x = max faces of the listed box elements: a quarter of each face to its corners
                area = m.ly / m.ny * m.lz / m.nz
                for a in (1, 2, 5, 6):
                    for c in range(3):
                        np.add.at(F[:, k], 3 * m.conn[p.elem_sets[it[1]], a] + c, it[4][c] * area / 4)
    return F


def _fixed_dofs(p):
    dpn = p.mesh.dpn
    return np.concatenate([dpn * p.node_sets[t[0][0]] + t[0][1] - 1 for t, _ in p.constraints])


def _static_planes(p, nu):
    m = p.mesh
    if m.elem_type == 4:
        n_tet, which = len(m.conn) // 6, np.repeat(np.arange(6), len(m.conn) // 6)
        mats = []
        for k in range(6):
            B, vol = _tet_b(m.coords[m.conn[k * n_tet]])
            mats.append(B.T @ _solid_c(nu) @ B * vol)
        A = _Planes(m.conn, (m.ny + 1) * (m.nz + 1), 3, p.E, np.stack(mats), which)
    else:
        K, _ = _hex_matrices((m.lx / m.nx, m.ly / m.ny, m.lz / m.nz), nu, m.elem_type == 81)
        A = _Planes(m.conn, (m.ny + 1) * (m.nz + 1), 3, p.E, K)
    A.add_diagonal(_fixed_dofs(p), 1e5 * A.largest())
    return A.factor()


def _tet_b(x):
    J = (x[1:] - x[0]).T
    g = np.concatenate([-np.ones((1, 3)), np.eye(3)]) @ np.linalg.inv(J)
    return _solid_b(g), np.linalg.det(J) / 6


def _exact_static(p, nu, tip=None):
    A = _static_planes(p, nu)
    f = torch.as_tensor(_loads(p), device=_device())
    u = A.solve(f)
    if tip is None:  # compliance
        return u, float((f * u).sum()), -A.energy(u, u)
    dl = torch.zeros(len(u), 1, dtype=torch.float64, device=u.device)
    dl[torch.as_tensor(np.asarray(tip[0], dtype=np.int64), device=u.device)] = tip[1]
    lam = A.solve(dl)
    return u, float((dl * u.sum(dim=1, keepdim=True)).sum()), -A.energy(lam, u.sum(dim=1, keepdim=True))


def _exact_newmark(A, M, f0, amp, dt, c_m):
    """Displacements [steps, n] of the reference's Newmark loop; A = K + c_m M + penalty."""
    c1, c2 = 1.0 / (dt * dt * (BETA - GAMMA)), dt * dt * (0.5 + BETA - GAMMA)
    u = torch.zeros_like(f0)
    a, up, vp, ap = u.clone(), u.clone(), u.clone(), u.clone()
    hist = []
    for w in amp:
        un = u + A.solve(float(w) * f0 - A.times(u) - M.times(a - c_m * u))
        an = c1 * (up - un + dt * vp + c2 * ap)
        vn = vp + dt * ((1 - GAMMA) * ap + GAMMA * an)
        up, vp, ap = un, vn, an
        u, a = un, c1 * (dt * vn + c2 * an)
        hist.append(un)
    return hist


def _dynamic_planes(conn, plane, dpn, E, rho, K, M, dt, fixed):
    c_m = -1.0 / (dt * dt * (BETA - GAMMA))
    A = _Planes(conn, plane, dpn, E, K)
    Mp = _Planes(conn, plane, dpn, rho, M)
    A.D += c_m * Mp.D
    A.U += c_m * Mp.U
    A.add_diagonal(fixed, 1e5 * A.largest())
    return A.factor(), Mp, c_m


def exact(case, seed):
    kind = case["kind"]
    if kind in ("learned", "train") or case.get("ny", 0) * case.get("nz", 0) * case.get("nx", 0) > 60000:
        return None  # a bandwidth of thousands over a hundred planes; a BF16 network
    if kind == "batch":
        inst = _batch_instances(case, seed)
        prob, node_ptr, elem_ptr = combine(inst)
        u, L, g = np.zeros((4, 3 * prob.mesh.n_nodes)), 0.0, np.zeros(prob.mesh.n_elems)
        for k, p in enumerate(inst):
            ui, Li, gi = _exact_static(p, float(p.nu[0]))
            u[:, 3 * node_ptr[k]:3 * node_ptr[k] + len(ui)] = _host(ui.T)
            g[elem_ptr[k]:elem_ptr[k + 1]] = _host(gi)
            L += Li
        return {"u": u, "L": np.array([L]), "dLdE": g}
    p = _problem(case, seed)
    m, nu = p.mesh, float(p.nu[0])
    if kind == "oneshot":
        u = _static_planes(p, nu).solve(torch.as_tensor(_loads(p), device=_device()))
        u = _host(u)[:, 0]
        n_tet, eps, vol = len(m.conn) // 6, np.zeros((len(m.conn), 6)), np.zeros(len(m.conn))
        for k in range(6):
            sel = slice(k * n_tet, (k + 1) * n_tet)
            B, v = _tet_b(m.coords[m.conn[k * n_tet]])
            ue = u.reshape(-1, 3)[m.conn[sel]].reshape(n_tet, 12)
            eps[sel], vol[sel] = ue @ B.T, v
        return {"u": u[None], "strain": eps, "stress": eps @ _solid_c(nu) * p.E[:, None], "volume": vol}
    if kind == "job":
        u, L, g = _exact_static(p, nu, (3 * p.node_sets["tip"] + 2, 1.0))
        g = _host(g)
        return {"u": _host(u.T), "L": np.array([L]), "dLdE": g,
                "dLdD": np.array([g[p.elem_sets[name]].sum() for name, _ in p.design_vars])}
    if kind == "multicase":
        return {"u": _host(_exact_static(p, nu)[0].T)}
    if kind in ("design", "brickim"):
        tip = (3 * p.node_sets["tip"] + 2, p.objective[3]) if kind == "brickim" else None
        u, L, g = _exact_static(p, nu, tip)
        return {"u": _host(u.T), "L": np.array([L]), "dLdE": _host(g)}
    if kind == "newmark":
        h = m.lx / m.nx
        K, M = _shell_matrices(h, h, nu, float(p.thickness[0]))
        A, Mp, c_m = _dynamic_planes(m.conn, m.ny + 1, 6, p.E, p.rho, K, M, PLATE_DT, _fixed_dofs(p))
        hist = _exact_newmark(A, Mp, torch.as_tensor(_loads(p), device=_device()), _plate_load(case), PLATE_DT, c_m)
        probe = 6 * int(p.node_sets["centre"][0]) + 2
        return {"history": np.array([float(h[probe, 0]) for h in hist]), "u": _host(hist[-1])[:, 0]}
    K, M = _hex_matrices((m.lx / m.nx, m.ly / m.ny, m.lz / m.nz), nu)
    plane = (m.ny + 1) * (m.nz + 1)
    if kind == "transient":
        dt = BEAM_DT
        A, Mp, c_m = _dynamic_planes(m.conn, plane, 3, p.E, p.rho, K, M, dt, _fixed_dofs(p))
        hist = _exact_newmark(A, Mp, torch.as_tensor(_loads(p), device=_device()), _transient_load(case), dt, c_m)
        dofs = 3 * p.node_sets["tip"] + 2
        w = torch.zeros_like(hist[0])
        w[torch.as_tensor(dofs.astype(np.int64), device=w.device)] = 1.0 / len(dofs)
        au = 1.0 / (dt * dt * (BETA - GAMMA))  # d a / d u_prev of the corrector, and its other factors
        av, aa = au * dt, au * dt * dt * (0.5 + BETA - GAMMA)
        c3, c4 = dt * (1 - GAMMA), 1.0 / (dt * (BETA - GAMMA))
        L, g = 0.0, 0.0
        lam = v_adj = a_adj = None
        for u in reversed(hist):
            L += float((w * u).sum())
            du, dv, da = w, torch.zeros_like(w), torch.zeros_like(w)
            if lam is not None:
                mu = Mp.times(lam)
                du = w - au * mu + au * a_adj
                da = -aa * mu + aa * a_adj + c3 * v_adj
                dv = -av * mu + c4 * a_adj + v_adj
            v_adj, a_adj = dv, da + dt * GAMMA * dv
            lam = A.solve(du - au * a_adj)
            g = g - A.energy(lam, u)
        return {"history": np.array([float(u[int(dofs[0]), 0]) for u in hist]), "u": _host(hist[-1])[:, 0],
                "L": np.array([L]), "dLdE": _host(g)}
    # modal: subspace iteration on the shift-free inverse
    A = _static_planes(p, nu)
    D = np.zeros(m.n_dof)
    for a in range(8):
        for c in range(3):
            np.add.at(D, 3 * m.conn[:, a] + c, p.rho * M[3 * a + c].sum())
    Dt, n = torch.as_tensor(D, device=_device())[:, None], case["modes"]
    X = torch.as_tensor(np.random.default_rng(0).standard_normal((m.n_dof, n + 12)), device=_device())
    lam = None
    for _ in range(80):
        X = torch.linalg.qr(A.solve(Dt * X, refine=0))[0]
        small_m = X.T @ (Dt * X)
        R = torch.linalg.cholesky(small_m)
        T = torch.linalg.solve_triangular(R, X.T @ A.times(X), upper=False)
        T = torch.linalg.solve_triangular(R, T.T, upper=False)
        new, S = torch.linalg.eigh(0.5 * (T + T.T))
        X = X @ torch.linalg.solve_triangular(R.T, S, upper=True)
        done = lam is not None and float((new[:n] / lam[:n] - 1).abs().max()) < 1e-13
        lam = new
        if done:
            break
    lam = _host(lam[:n])
    return {"eigenvalues": lam, "frequencies": np.sqrt(lam) / (2 * math.pi), "mass": D}
