"""The V-cycle's fused tail against one launch per level and step: the same sums in
the same order, so the same bits, for tails of two to five levels, levels with
fewer rows than CTAs, one row a CTA and the most that fit, thin and odd blocks, and
up to four right-hand sides at once (chunks of four and the rest)."""
import numpy as np
import pytest

from asend3d_gb300 import _lib
from asend3d_gb300.mesh import block_hex8
from asend3d_gb300.solver import GpuSolver, Problem

pytestmark = pytest.mark.gpu


def bar(dims, cases=1, seed=4):
    nx, ny, nz = dims
    rng = np.random.default_rng(seed)
    m = block_hex8(nx, ny, nz, 0.1 * nx, 0.1 * ny, 0.1 * nz)
    p = Problem(m, 70e9 * np.exp(0.3 * rng.standard_normal(m.n_elems)), np.full(m.n_elems, 0.3))
    p.add_node_set("xMin", m.nodes_in_range(xr=(-1e-9, 1e-9)))
    p.fix_displacement("xMin")
    end = m.nodes_in_range(xr=(0.1 * nx - 1e-9, 1e9))
    p.add_node_set("end", end)
    for k in range(cases):
        p.add_nodal_force("end", [10.0 * k, 3.0, -100.0 / len(end)], case=k)
    return p


@pytest.mark.parametrize("dims", [(25, 12, 7), (80, 3, 3), (18, 18, 17), (37, 1, 21), (64, 24, 20), (30, 30, 30)])
def test_vcycle_bits(gpu_lib, dims):
    g = GpuSolver(bar(dims))
    g.assemble(64)
    rng = np.random.default_rng(2)
    for _ in range(2):
        b = rng.standard_normal(g.n_dof).astype(np.float32)
        z = []
        for tail in (False, True):
            g.mg_set_fused_tail(tail)
            z.append(g.mg_vcycle(b))
        assert np.all(np.isfinite(z[0])) and np.array_equal(z[0], z[1])
    assert g.mg_levels > 2
    g.close()


@pytest.mark.parametrize("cases", [2, 5])
@pytest.mark.parametrize("overlap", [False, True])
def test_solve_bits(gpu_lib, cases, overlap):
    g = GpuSolver(bar((40, 12, 13), cases))
    g.assemble(64)
    g.set_launch_overlap(overlap)
    u = []
    for tail in (False, True):
        g.mg_set_fused_tail(tail)
        x, rc, _ = g.static_solve(method=_lib.METHOD_SPLIT, precond=_lib.PC_MG, rel_tol=1e-9)
        assert rc == 0
        u.append(x)
    assert np.array_equal(u[0], u[1])
    g.close()
