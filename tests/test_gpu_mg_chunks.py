"""Short last chunks of the multigrid CG: the same bits and iteration counts whatever
the chunk length (a chunk of one iteration never has a short stretch), and the
iteration cap still ends a solve that it cuts off."""
import numpy as np
import pytest

from asend3d_gb300 import _lib
from asend3d_gb300.mesh import block_hex8
from asend3d_gb300.solver import GpuSolver, Problem

pytestmark = pytest.mark.gpu


def bar(dims, cases):
    nx, ny, nz = dims
    rng = np.random.default_rng(6)
    m = block_hex8(nx, ny, nz, 0.1 * nx, 0.1 * ny, 0.1 * nz)
    p = Problem(m, 70e9 * np.exp(0.3 * rng.standard_normal(m.n_elems)), np.full(m.n_elems, 0.3))
    p.add_node_set("xMin", m.nodes_in_range(xr=(-1e-9, 1e-9)))
    p.fix_displacement("xMin")
    end = m.nodes_in_range(xr=(0.1 * nx - 1e-9, 1e9))
    p.add_node_set("end", end)
    for k in range(cases):
        p.add_nodal_force("end", [10.0 * k, 3.0, -100.0 / len(end)], case=k)
    return p


@pytest.mark.parametrize("dims,cases", [((6, 6, 6), 1), ((30, 9, 7), 3)])
@pytest.mark.parametrize("method", [_lib.METHOD_SPLIT, _lib.METHOD_FP64])
def test_same_bits_for_every_chunk_length(gpu_lib, dims, cases, method):
    g = GpuSolver(bar(dims, cases))
    g.assemble(64)
    ref = None
    for graph_iters in (1, 2, 3, 4, 5, 8, 16, 40):
        u, rc, st = g.static_solve(method=method, precond=_lib.PC_MG, rel_tol=1e-9, graph_iters=graph_iters)
        assert rc == 0
        if ref is None:
            ref = u, st["iterations"]
        assert np.array_equal(u, ref[0]) and st["iterations"] == ref[1], graph_iters
    g.close()


@pytest.mark.parametrize("graph_iters", [2, 8])
def test_iteration_cap(gpu_lib, graph_iters):
    g = GpuSolver(bar((30, 9, 7), 1))
    g.assemble(64)
    _, rc, st = g.static_solve(method=_lib.METHOD_SPLIT, precond=_lib.PC_MG, rel_tol=1e-10, graph_iters=graph_iters,
                               max_iter=8)
    assert rc == 1 and st["iterations"] == 8
    g.close()
