"""A coarse level's values, smoother blocks and eigenvalue estimates against a
NumPy Galerkin product, for blocks of one slice and several, odd and even sides, a
side of one cell, axes that are and are not coarsened, and a stack.

Checked through the guaranteed bound max_n ||(D^-1 A)_n||_inf of a level, which
takes every value of its rows, and through the power iteration from its hashed
start vector.  Rows on the clamped end carry a penalty 1e5 times the largest stiffness:
their rows of D^-1 A are the identity's but for 1e-5 or less, the size of the
estimate's tolerance 1e-4; the bound is reached on free rows, whose values are FP32
sums of at most 64 rounded terms, each block row adding up 81 of them: 1e-5."""
import numpy as np
import pytest
import scipy.sparse as sp

from asend3d_gb300.mesh import block_hex8
from asend3d_gb300.solver import GpuSolver, Problem, combine

pytestmark = pytest.mark.gpu

POWER_STEPS = 10


def bar(dims, fixed=True, elem_type=8, seed=3):
    nx, ny, nz = dims
    rng = np.random.default_rng(seed)
    m = block_hex8(nx, ny, nz, 0.1 * nx, 0.08 * ny, 0.09 * nz)
    m.elem_type = elem_type
    p = Problem(m, 70e9 * np.exp(0.4 * rng.standard_normal(m.n_elems)), np.full(m.n_elems, 0.3))
    p.add_node_set("xMin", m.nodes_in_range(xr=(-1e-9, 1e-9)))
    if fixed:
        p.fix_displacement("xMin")
    p.add_node_set("end", m.nodes_in_range(xr=(0.1 * nx - 1e-9, 1e9)))
    p.add_nodal_force("end", [0.0, 0.0, -1.0])
    return p


def axis_map(nf, nc):
    P = np.zeros((nf + 1, nc + 1))
    at = [m if nc == nf else min(2 * m, nf) for m in range(nc + 1)]
    for m in range(nc):
        for f in range(at[m], at[m + 1] + 1):
            t = (f - at[m]) / (at[m + 1] - at[m])
            P[f, m], P[f, m + 1] = 1 - t, t
    P[at[nc], nc] = 1.0
    return P


def reference(dims, levels, elem_type=8):
    """Bound and power estimate of every level but the coarsest."""
    g = GpuSolver(bar(dims, fixed=False, elem_type=elem_type))
    g.assemble(64)
    rp, col, val = g.csr(0)
    g.close()
    n = (dims[0] + 1) * (dims[1] + 1) * (dims[2] + 1)
    A = sp.csr_matrix((val, col, rp), shape=(3 * n, 3 * n))
    out = []
    for f, c in zip(levels[:-1], levels[1:]):
        P = sp.kron(sp.kron(sp.kron(axis_map(f[0], c[0]), axis_map(f[1], c[1])), axis_map(f[2], c[2])), sp.eye(3)).tocsr()
        A = (P.T @ A @ P).tocsr()
        if c == levels[-1]:
            break
        nn = A.shape[0] // 3
        B = A.tobsr((3, 3))
        B.sort_indices()
        D = np.zeros((nn, 3, 3))
        for r in range(nn):
            k = B.indptr[r] + np.searchsorted(B.indices[B.indptr[r]:B.indptr[r + 1]], r)
            D[r] = B.data[k]
        Di = sp.bsr_matrix((np.linalg.inv(D), np.arange(nn), np.arange(nn + 1)), shape=A.shape)
        S = (Di @ A).tocsr()
        free = np.repeat(np.arange(nn) >= (c[1] + 1) * (c[2] + 1), 3)
        bound = np.asarray(abs(S).sum(axis=1)).ravel()[free].max()
        v = np.arange(1, 3 * nn + 1, dtype=np.uint32)
        for sh, mul in ((16, 0x7feb352d), (15, 0x846ca68b), (16, 1)):
            v ^= v >> np.uint32(sh)
            v = (v * np.uint64(mul)).astype(np.uint32) if mul > 1 else v
        x = (v >> np.uint32(8)) * (2.0 / 16777216.0) - 1.0
        nrm = 1.0
        for _ in range(POWER_STEPS):
            x = x / nrm
            x = np.where(free, S @ x, x)
            nrm = np.linalg.norm(x)
        out.append((bound, nrm))
    return out


def infos(g):
    return [g.mg_level_info(l) for l in range(g.mg_levels)]


@pytest.mark.parametrize("dims", [(14, 6, 5), (33, 11, 3), (40, 16, 16), (21, 1, 9)])
@pytest.mark.parametrize("elem_type", [8, 81])
def test_level_values(gpu_lib, dims, elem_type):
    g = GpuSolver(bar(dims, elem_type=elem_type))
    g.assemble(64)
    g.mg_vcycle(np.ones(g.n_dof, np.float32))
    info = infos(g)
    g.close()
    assert len(info) > 1
    for l, (bound, est) in enumerate(reference(dims, [i["dims"] for i in info], elem_type), start=1):
        assert info[l]["lambda_bound"] == pytest.approx(bound, rel=1e-5)
        assert info[l]["lambda_est"] == pytest.approx(est, rel=1e-4)


def test_stack_values(gpu_lib):
    members = [(30, 7, 9), (28, 7, 9)]
    lone = []
    for k, d in enumerate(members):
        g = GpuSolver(bar(d, seed=k))
        g.assemble(64)
        g.mg_vcycle(np.ones(g.n_dof, np.float32))
        lone.append(infos(g))
        g.close()
    p, inst, _ = combine([bar(d, seed=k) for k, d in enumerate(members)])
    g = GpuSolver(p, instances=inst, blocks=members)
    g.assemble(64)
    g.mg_vcycle(np.ones(g.n_dof, np.float32))
    info = infos(g)
    g.close()
    assert len(info) == len(lone[0]) == len(lone[1]) > 2
    for l in range(1, len(info) - 1):
        assert info[l]["lambda_bound"] == pytest.approx(max(x[l]["lambda_bound"] for x in lone), rel=1e-6)
