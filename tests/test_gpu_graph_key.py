"""Captured multigrid iterations after a change of the assembly's precision: the
matrix-free products of a pair assembly (48) whose FP64 values were asked for
take that operator's patterns, whatever was captured before, and the same the
other way round."""
import numpy as np
import pytest

from asend3d_gb300 import _lib
from asend3d_gb300.mesh import block_hex8
from asend3d_gb300.solver import GpuSolver, Problem

pytestmark = pytest.mark.gpu


def bar():
    rng = np.random.default_rng(8)
    m = block_hex8(23, 6, 5, 2.3, 0.42, 0.4)
    p = Problem(m, 70e9 * np.exp(0.3 * rng.standard_normal(m.n_elems)), np.full(m.n_elems, 0.3))
    p.add_node_set("xMin", m.nodes_in_range(xr=(-1e-9, 1e-9)))
    p.fix_displacement("xMin")
    end = m.nodes_in_range(xr=(2.3 - 1e-9, 1e9))
    p.add_node_set("end", end)
    p.add_nodal_force("end", [10.0, 3.0, -100.0 / len(end)])
    return p


@pytest.mark.parametrize("first,second", [(64, 48), (48, 64)])
def test_patterns_follow_the_assembly(gpu_lib, first, second):
    """The second solve reuses the first one's graphs, or (another chunk length
    first, which does not change a result) captures its own: the same bits."""
    u = []
    for chunk in (8, 7):
        g = GpuSolver(bar())
        for precision, graph_iters in ((first, chunk), (second, 8)):
            g.assemble(precision)
            g.csr(0)  # FP64 values
            x, rc, _ = g.static_solve(method=_lib.METHOD_SPLIT, precond=_lib.PC_MG, rel_tol=1e-10, max_iter=500,
                                      graph_iters=graph_iters)
            assert rc == 0
        u.append(x[0])
        g.close()
    assert np.array_equal(u[0], u[1])
