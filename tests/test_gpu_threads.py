"""A context per host thread: two models of different sizes solved at the same
time, whose launches of the same kernel take different amounts of shared memory.
Every Jacobi solve gives the bits that it gives alone; a multigrid solve (whose
eigenvalue estimates start from the previous set-up's vectors) meets its tolerance
in the host's residual, with the rounding of the host's product (81 terms a row)."""
import threading

import numpy as np
import pytest

from asend3d_gb300 import _lib
from asend3d_gb300.mesh import block_hex8
from asend3d_gb300.solver import GpuSolver, Problem

pytestmark = pytest.mark.gpu


def bar(dims):
    nx, ny, nz = dims
    rng = np.random.default_rng(4)
    m = block_hex8(nx, ny, nz, 0.1 * nx, 0.1 * ny, 0.1 * nz)
    p = Problem(m, 70e9 * np.exp(0.3 * rng.standard_normal(m.n_elems)), np.full(m.n_elems, 0.3))
    p.add_node_set("xMin", m.nodes_in_range(xr=(-1e-9, 1e-9)))
    p.fix_displacement("xMin")
    p.add_load_vector(1000.0 * rng.standard_normal(m.n_dof))
    return p


def met(csr, f, u, rel_tol):
    rp, col, val = csr
    r = f - np.add.reduceat(val * u[col], rp[:-1])
    size = np.add.reduceat(np.abs(val * u[col]), rp[:-1])
    return np.linalg.norm(r) <= rel_tol * np.linalg.norm(f) + 2 * 81 * np.finfo(float).eps * np.linalg.norm(size)


# loose tolerances: solves of a few launches, back to back
@pytest.mark.parametrize("kw,sizes", [
    (dict(method=_lib.METHOD_FP64, precond=_lib.PC_JACOBI, rel_tol=0.3), [(20, 4, 4), (57, 13, 11)]),
    (dict(method=_lib.METHOD_MIXED, precond=_lib.PC_BLOCK, rel_tol=0.3), [(12, 4, 4), (40, 13, 11)]),
    (dict(method=_lib.METHOD_SPLIT, precond=_lib.PC_MG, rel_tol=0.3), [(9, 3, 3), (9, 12, 60)])])
def test_two_contexts(gpu_lib, kw, sizes, solves=800):
    def work(g, n, out):
        try:
            for _ in range(n):
                g.assemble(64)
                u, rc, _ = g.static_solve(**kw)
                assert rc == 0
                out.append(u[0])
        except Exception as e:  # handed to the test's thread
            out.append(e)

    solvers = [GpuSolver(bar(s)) for s in sizes]
    alone = []
    for g in solvers:
        one = []
        work(g, 1, one)
        alone.append(one[0])
    results = [[], []]
    threads = [threading.Thread(target=work, args=(g, solves, r)) for g, r in zip(solvers, results)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for r in results:
        assert not [e for e in r if isinstance(e, Exception)]
    for g, r, a in zip(solvers, results, alone):
        assert len(r) == solves
        if kw["precond"] == _lib.PC_MG:
            csr, f = g.csr(0), g.load_vector()
            assert all(met(csr, f, u, kw["rel_tol"]) for u in r)
        else:
            assert all(np.array_equal(u, a) for u in r)
        g.close()
