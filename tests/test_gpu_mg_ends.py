"""Load cases of one multigrid solve end apart: a case that turns non-finite or
meets the iteration cap leaves the others to converge, as each does alone.
Solutions to 1e-8 in the residual (which the mixed method reaches on a cube): checked
in the host's residual with the rounding of its own product, n_row eps || |A| |u| ||
(n_row = 81)."""
import numpy as np
import pytest

from asend3d_gb300 import _lib
from asend3d_gb300.mesh import block_hex8
from asend3d_gb300.solver import GpuSolver, Problem, combine

pytestmark = pytest.mark.gpu

TOL = 1e-8


def bar(loads, dims=(8, 8, 8), seed=3):
    nx, ny, nz = dims
    rng = np.random.default_rng(seed)
    m = block_hex8(nx, ny, nz, 0.1 * nx, 0.1 * ny, 0.1 * nz)
    p = Problem(m, 70e9 * np.exp(0.3 * rng.standard_normal(m.n_elems)), np.full(m.n_elems, 0.3))
    p.add_node_set("xMin", m.nodes_in_range(xr=(-1e-9, 1e-9)))
    p.fix_displacement("xMin")
    for k, f in enumerate(loads):
        p.add_load_vector(f(m, np.random.default_rng(100 + k)), case=k)
    return p


def rough(m, rng):
    return 1000.0 * rng.standard_normal(m.n_dof)


def bend(m, rng):
    f = np.zeros(m.n_dof)
    f[3 * np.flatnonzero(m.coords[:, 0] > m.coords[:, 0].max() - 1e-9) + 2] = -100.0
    return f


def too_large(m, rng):
    return 1e200 * rng.standard_normal(m.n_dof)  # |f|^2 overflows


def met(g, f, u):
    rp, col, val = g.csr(0)
    r = f - np.add.reduceat(val * u[col], rp[:-1])
    size = np.add.reduceat(np.abs(val * u[col]), rp[:-1])
    return np.linalg.norm(r) <= TOL * np.linalg.norm(f) + 2 * 81 * np.finfo(float).eps * np.linalg.norm(size)


@pytest.mark.parametrize("method", [_lib.METHOD_SPLIT, _lib.METHOD_FP64])
@pytest.mark.parametrize("bad", [0, 2])
def test_non_finite_case(gpu_lib, method, bad):
    loads = [rough, bend, rough, bend, rough]
    loads[bad] = too_large
    p = bar(loads)
    g = GpuSolver(p)
    g.assemble(64)
    u, rc, _ = g.static_solve(method=method, precond=_lib.PC_MG, rel_tol=TOL, max_iter=300)
    assert rc == 2
    for k in range(5):
        if k != bad:
            assert met(g, g.load_vector(k), u[k]), k
    g.close()


@pytest.mark.parametrize("method", [_lib.METHOD_SPLIT, _lib.METHOD_MIXED])
def test_capped_case(gpu_lib, method):
    """The cap lies above the shorter case's iterations, at or below the longer one's."""
    kw = dict(method=method, precond=_lib.PC_MG, rel_tol=TOL)

    def solve(loads, **extra):
        g = GpuSolver(bar(loads))
        g.assemble(64)
        u, rc, st = g.static_solve(**kw, **extra)
        ok = [met(g, g.load_vector(k), u[k]) for k in range(len(loads))]
        g.close()
        return rc, st["iterations"], ok

    its = [solve([f])[1] for f in (rough, bend)]
    assert its[0] < its[1]
    cap = its[0] + 1
    assert solve([rough], max_iter=cap)[0] == 0
    assert solve([rough, bend], max_iter=cap)[2][0]
    assert solve([bend, rough], max_iter=cap)[2][1]


def test_non_finite_case_of_a_stack(gpu_lib):
    dims = [(20, 4, 4), (33, 9, 7)]
    loads = [rough, too_large, bend]
    p, ptr, _ = combine([bar(loads, d, seed=i) for i, d in enumerate(dims)])
    g = GpuSolver(p, instances=ptr, blocks=dims)
    g.assemble(64)
    u, rc, _ = g.static_solve(method=_lib.METHOD_SPLIT, precond=_lib.PC_MG, rel_tol=TOL, max_iter=300)
    assert rc == 2
    for k in (0, 2):
        assert met(g, g.load_vector(k), u[k]), k
    g.close()
