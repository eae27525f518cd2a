"""Pieces of the multigrid set-up and of the class gradient, each at the sizes
where its kernel changes shape.

Coarsest inverse: a block of at most 256 DOF is its own coarsest level, so the
preconditioner is the FP32 inverse itself.  CG then gains at least the factor
1 / (kappa eps32) a step; these blocks' scaled condition numbers are below 1e4
(short beams), so 6e-4 a step and 1e-10 within 4 steps: at most 5 are asked,
one for the confirmation.

Class gradient of brickIM: the same FP64 contraction as the oracle's on the
same fields; 576 products a side, element strains some 1e-2 of the element's
relative displacements, so 1e3 x 576 x 1.1e-16 < 1e-10."""
import numpy as np
import pytest

from asend3d_gb300 import _lib
from asend3d_gb300.mesh import block_hex8
from asend3d_gb300.solver import GpuSolver, Problem

pytestmark = pytest.mark.gpu


def block(nx, ny, nz, elem_type=8, distort=0.0, seed=5):
    rng = np.random.default_rng(seed)
    m = block_hex8(nx, ny, nz, 0.1 * nx, 0.1 * ny, 0.1 * nz)
    m.elem_type = elem_type
    if distort:
        m.coords = m.coords + rng.uniform(-distort, distort, m.coords.shape)
    p = Problem(m, 70e9 * np.exp(0.3 * rng.standard_normal(m.n_elems)), np.full(m.n_elems, 0.3))
    p.add_node_set("fixed", m.node_id(0, *np.meshgrid(np.arange(ny + 1), np.arange(nz + 1), indexing="ij")).ravel())
    p.fix_displacement("fixed")
    tip = np.array([m.node_id(nx, ny, nz)])
    p.add_node_set("tip", tip)
    p.add_nodal_force("tip", [300.0, 200.0, -1000.0])
    return p


# 24, 54, 96, 99 (a panel and a row more), 192, 243 and 252 DOF
@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 2, 1), (3, 3, 1), (2, 2, 2), (3, 3, 3), (8, 2, 2), (6, 3, 2)])
@pytest.mark.parametrize("method", [_lib.METHOD_FP64, _lib.METHOD_SPLIT])
def test_coarsest_inverse(gpu_lib, dims, method):
    g = GpuSolver(block(*dims))
    g.assemble(64)
    u, rc, st = g.static_solve(method=method, precond=_lib.PC_MG, rel_tol=1e-10)
    assert rc == 0 and g.mg_levels == 1 and st["iterations"] <= 5
    g.close()


@pytest.mark.parametrize("distort", [0.0, 0.01])
def test_brickim_class_gradient(gpu_lib, oracle_lib, distort):
    p = block(5, 3, 2, elem_type=81, distort=distort)
    g = GpuSolver(p)
    g.assemble(64)
    kw = dict(method=_lib.METHOD_FP64, precond=_lib.PC_JACOBI, rel_tol=1e-12)
    u, rc, _ = g.static_solve(**kw)
    _, grad, rc2, _ = g.adjoint_gradient(**kw)
    assert rc == 0 and rc2 == 0
    ref = oracle_lib.Oracle(p).adjoint(u[0], lam=u[0])[0]
    assert np.linalg.norm(grad - ref) <= 1e-10 * np.linalg.norm(ref)
    g.close()
