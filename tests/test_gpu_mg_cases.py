"""Multigrid CG over several load cases at once (a chunk of up to four and a
remainder) and the FP64 product with lanes.

A case's vectors, scalars and sums are its own, so a solve of several cases is
bit-identical to solves of each case alone in a new context (the coarse levels'
eigenvalue estimates start from the previous assembly's vectors in an old one).
Solutions of the FP64 and the split method to 1e-10 in the residual carry errors
of that order (end-loaded bars): they agree to 1e-9."""
import numpy as np
import pytest

from asend3d_gb300 import _lib
from asend3d_gb300.mesh import block_hex8
from asend3d_gb300.solver import GpuSolver, Problem, combine

pytestmark = pytest.mark.gpu


def bar(dims, cases, seed=2):
    nx, ny, nz = dims
    rng = np.random.default_rng(seed)
    m = block_hex8(nx, ny, nz, 0.1 * nx, 0.08 * ny, 0.09 * nz)
    p = Problem(m, 70e9 * np.exp(0.3 * rng.standard_normal(m.n_elems)), np.full(m.n_elems, 0.3))
    p.add_node_set("xMin", m.nodes_in_range(xr=(-1e-9, 1e-9)))
    p.fix_displacement("xMin")
    end = m.nodes_in_range(xr=(0.1 * nx - 1e-9, 1e9))
    p.add_node_set("end", end)
    for k in cases:
        p.add_nodal_force("end", 1000.0 * np.random.default_rng(k).standard_normal(3) / len(end), case=len(p.loads))
    return p


def solve(p, method, inst=None, blocks=None, precision=48):
    g = GpuSolver(p, instances=inst, blocks=blocks)
    g.assemble(precision)
    u, rc, st = g.static_solve(method=method, precond=_lib.PC_MG, rel_tol=1e-10, max_iter=500)
    assert rc == 0 and st["n_rhs"] == len(p.loads)
    g.close()
    return u


@pytest.mark.parametrize("method", [_lib.METHOD_SPLIT, _lib.METHOD_FP64])
@pytest.mark.parametrize("dims,cases", [((3, 2, 2), 2), ((24, 7, 6), 5), ((40, 16, 16), 4)])
def test_cases_are_independent(gpu_lib, dims, cases, method):
    together = solve(bar(dims, range(cases)), method)
    for k in range(cases):
        assert np.array_equal(together[k], solve(bar(dims, [k]), method)[0])


def test_stack_cases_are_independent(gpu_lib):
    dims = [(20, 4, 4), (33, 9, 7), (8, 3, 5)]

    def stack(cases):
        return combine([bar(d, cases, seed=i) for i, d in enumerate(dims)])[:2]

    p, ptr = stack(range(5))
    together = solve(p, _lib.METHOD_SPLIT, ptr, dims)
    for k in range(5):
        p, ptr = stack([k])
        assert np.array_equal(together[k], solve(p, _lib.METHOD_SPLIT, ptr, dims)[0])


# rows that take eight lanes (below 38,912), one more block of rows, and one thread
@pytest.mark.parametrize("dims", [(5, 4, 4), (50, 12, 11), (60, 24, 25)])
def test_fp64_product_with_lanes(gpu_lib, dims):
    p = bar(dims, [0])
    u64 = solve(p, _lib.METHOD_FP64, precision=64)[0]
    us = solve(p, _lib.METHOD_SPLIT, precision=64)[0]
    assert np.linalg.norm(u64 - us) <= 1e-9 * np.linalg.norm(us)
