"""The one-launch PCG with its operator in shared memory (k_resident.cu) at the
edges of its layout: fewer rows than a CTA takes, lanes of a row from 16 down
to 1, values on chip and streamed, one to five right-hand sides (a chunk of
four and a remainder), point and nodal-block Jacobi, warm starts, the cap.

The operators are those of a time step (stiffness and mass), on which the mixed
method converges too.  Tolerances: a converged solve has ||f - A u|| <= 1e-10
||f|| in the library's FP64 evaluation; it and the host's each differ from the
exact product by at most n_row eps || |A| |u| || (n_row <= 81), which is computed
and added.  Newmark histories of two runs of the same recurrences, each step
solved to 1e-12: 1e-9 (the increments' errors over some twenty steps)."""
import numpy as np
import pytest

from asend3d_gb300 import _lib, configs
from asend3d_gb300.mesh import block_hex8, block_tet4
from asend3d_gb300.solver import GpuSolver, Problem

pytestmark = pytest.mark.gpu


def residual_and_bound(g, f, u, rel_tol=1e-10):
    """||f - A u|| in FP64 on the host, and what it may be."""
    rp, col, val = g.csr(0)
    r = f - np.add.reduceat(val * u[col], rp[:-1])
    size = np.add.reduceat(np.abs(val * u[col]), rp[:-1])
    eps = np.finfo(np.float64).eps
    return np.linalg.norm(r), rel_tol * np.linalg.norm(f) + 2 * 81 * eps * np.linalg.norm(size)


def model(mesh, cases, seed=3):
    rng = np.random.default_rng(seed)
    p = Problem(mesh, 70e9 * np.exp(0.3 * rng.standard_normal(mesh.n_elems)), np.full(mesh.n_elems, 0.3),
                np.full(mesh.n_elems, 2700.0))
    p.add_node_set("xMin", mesh.nodes_in_range(xr=(-1e-9, 1e-9)))
    p.fix_displacement("xMin")
    for k in range(cases):
        p.add_load_vector(1000.0 * rng.standard_normal(mesh.n_dof), case=k)
    return p


# 8 nodes (one CTA); 525 rows (T 16); 4,961 (T 16, several warps); 11,713 tet
# rows (T 8, short rows); 29,161 (192 rows a CTA: T 2, streamed values); 49,011
# (323 rows: T 1, one right-hand side only: five take the general kernels)
@pytest.mark.parametrize("dims,tet,cases", [((1, 1, 1), False, 1), ((20, 4, 4), False, 5), ((60, 8, 8), False, 3),
                                            ((52, 12, 16), True, 2), ((40, 26, 26), False, 1),
                                            ((40, 26, 26), False, 2), ((60, 25, 30), False, 1)])
@pytest.mark.parametrize("method", [_lib.METHOD_FP64, _lib.METHOD_MIXED])
@pytest.mark.parametrize("precond", [_lib.PC_JACOBI, _lib.PC_BLOCK])
def test_residual_is_met(gpu_lib, dims, tet, cases, method, precond):
    m = (block_tet4 if tet else block_hex8)(*dims, 0.1 * dims[0], 0.1 * dims[1], 0.1 * dims[2])
    p = model(m, cases)
    g = GpuSolver(p)
    g.assemble(64, dynamic=True, dt=2e-5)
    launches = g.kernel_launches
    u, rc, st = g.static_solve(method=method, precond=precond, rel_tol=1e-10, max_iter=20000)
    assert rc == 0 and st["iterations"] > 0
    if m.n_nodes < 32000 or cases == 1:  # one launch a chunk, and the preconditioner's
        assert g.kernel_launches - launches <= (cases + 3) // 4 + 1
    for k in range(cases):
        r, bound = residual_and_bound(g, g.load_vector(k), u[k])
        assert r <= bound
    # from the solution: nothing left to do
    u2, rc2, st2 = g.static_solve(u0=u, method=method, precond=precond, rel_tol=2e-10)
    assert rc2 == 0 and st2["iterations"] == 0 and np.array_equal(u2, u)
    g.close()


def test_cap_and_replacement(gpu_lib):
    g = GpuSolver(model(block_hex8(12, 4, 3, 3.0, 1.0, 1.0), 1))
    g.assemble(64)
    kw = dict(method=_lib.METHOD_FP64, precond=_lib.PC_JACOBI, rel_tol=1e-10)
    u, rc, st = g.static_solve(max_iter=10, graph_iters=4, **kw)
    assert rc == _lib.ASEND_MAX_ITER and st["iterations"] == 12  # whole chunks of graph_iters
    u, rc, st = g.static_solve(replace_every=5, **kw)
    assert rc == 0 and st["replacements"] >= st["iterations"] // 5
    r, bound = residual_and_bound(g, g.load_vector(0), u[0])
    assert r <= bound
    g.close()


@pytest.mark.parametrize("damping", [None, (3.0, 0.0, None), (3.0, 1e-6, None)])
@pytest.mark.parametrize("warm", [0, 2])
def test_newmark_loop_matches_stepwise(gpu_lib, damping, warm):
    """The time loop inside the kernel against the step-by-step loop (an
    untrained learned preconditioner falls back to point Jacobi step by step)."""
    p = model(block_hex8(10, 3, 2, 1.0, 0.3, 0.2), 1)
    p.damping = damping
    amp = np.sin(np.linspace(0.2, 3.0, 20))
    out = []
    for precond in (_lib.PC_JACOBI, _lib.PC_LEARNED):
        g = GpuSolver(p)
        g.assemble(dynamic=True, dt=2e-4)
        g.keep_history(3)
        hist, u, rc, st = g.newmark(amp, probe_dof=100, method=_lib.METHOD_FP64, precond=precond, rel_tol=1e-12,
                                    warm_start=warm)
        assert rc == 0 and st["iterations"] > 0 and st["rel_residual"] <= 1e-12
        out.append([hist, u] + [x for s in (1, 2, 20) for x in g.step_state(s, fields=3)])
        assert np.array_equal(g.step_state(20)[0], u)
        g.close()
    for a, b in zip(*out):
        assert np.linalg.norm(a - b) <= 1e-9 * np.linalg.norm(b)
