"""Four right-hand sides by one reading of a coarse level's values against one
solve each, the same bits, on a stack whose first coarse level has just more rows
than the warps of the persistent grid (77,824) and on one that has just fewer."""
import numpy as np
import pytest

from asend3d_gb300 import _lib
from asend3d_gb300.mesh import block_hex8
from asend3d_gb300.solver import GpuSolver, Problem, combine

pytestmark = pytest.mark.gpu


def bar(dims, cases, seed):
    nx, ny, nz = dims
    rng = np.random.default_rng(seed)
    m = block_hex8(nx, ny, nz, 0.1 * nx, 0.04 * ny, 0.04 * nz)  # x is not coarsened first
    p = Problem(m, 70e9 * np.exp(0.3 * rng.standard_normal(m.n_elems)), np.full(m.n_elems, 0.3))
    p.add_node_set("xMin", m.nodes_in_range(xr=(-1e-9, 1e-9)))
    p.fix_displacement("xMin")
    end = m.nodes_in_range(xr=(0.1 * nx - 1e-9, 1e9))
    p.add_node_set("end", end)
    for i, k in enumerate(cases):
        p.add_nodal_force("end", [10.0 * k, 3.0, -100.0 / len(end)], case=i)
    return p


# rows of the first coarse level: 2 x 45 x 30 x 30 and 2 x 42 x 30 x 30 (and padding)
@pytest.mark.parametrize("nx", [44, 41])
def test_same_bits(gpu_lib, nx):
    dims = [(nx, 58, 58), (nx, 58, 57)]

    def solve(cases):
        p, ptr, _ = combine([bar(d, cases, seed=i) for i, d in enumerate(dims)])
        g = GpuSolver(p, instances=ptr, blocks=dims)
        g.assemble(48)
        u, rc, _ = g.static_solve(method=_lib.METHOD_SPLIT, precond=_lib.PC_MG, rel_tol=1e-8)
        g.close()
        assert rc == 0
        return u

    together = solve(range(4))
    for k in range(4):
        assert np.array_equal(together[k], solve([k])[0])
