"""Launch overlap on and off (set_launch_overlap): the same bits from the
matrix-free products, the fused V-cycle tail and the FP64 kernels, on a block and
on a stack, several load cases, two assemblies one after the other."""
import numpy as np
import pytest

from asend3d_gb300 import _lib
from asend3d_gb300.mesh import block_hex8
from asend3d_gb300.solver import GpuSolver, Problem, combine

pytestmark = pytest.mark.gpu


def bar(dims, seed=5):
    nx, ny, nz = dims
    rng = np.random.default_rng(seed)
    m = block_hex8(nx, ny, nz, 0.1 * nx, 0.1 * ny, 0.1 * nz)
    p = Problem(m, 70e9 * np.exp(0.3 * rng.standard_normal(m.n_elems)), np.full(m.n_elems, 0.3))
    p.add_node_set("xMin", m.nodes_in_range(xr=(-1e-9, 1e-9)))
    p.fix_displacement("xMin")
    for k in range(3):
        p.add_load_vector(1000.0 * rng.standard_normal(m.n_dof), case=k)
    return p


@pytest.mark.parametrize("method,precision", [(_lib.METHOD_SPLIT, 48), (_lib.METHOD_SPLIT, 64), (_lib.METHOD_FP64, 64)])
@pytest.mark.parametrize("stack", [False, True])
def test_same_bits(gpu_lib, method, precision, stack):
    dims = [(20, 4, 4), (33, 9, 7), (8, 3, 5)]
    out = []
    for overlap in (False, True):
        p, ptr, _ = combine([bar(d, seed=i) for i, d in enumerate(dims)]) if stack else (bar((44, 12, 11)), None, None)
        g = GpuSolver(p, instances=ptr, blocks=dims if stack else None)
        g.set_launch_overlap(overlap)
        for scale in (1.0, 1.3):
            g.set_modulus(scale * p.E)
            g.assemble(precision)
            u, rc, st = g.static_solve(method=method, precond=_lib.PC_MG, rel_tol=1e-10, max_iter=500)
            assert rc == 0
            out.append((u, st["iterations"]))
        g.close()
    for (u, its), (v, its_v) in zip(out[:2], out[2:]):
        assert np.array_equal(u, v) and its == its_v
