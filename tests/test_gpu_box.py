"""Matrix-free finest-level products (k_box.cu) against the assembled ones on the
same operator, at the edges of their layout: a plane inside one CTA, several
segments a plane, one plane a CTA, odd sizes, the largest and the first refused
nz, both hex types, stacks with padding nodes.

A constraint between two neighbouring nodes with coefficients 1e-9 (penalty
1e-13 of the largest stiffness) leaves the operator as it is but not diagonal in
its penalties, which is the assembled path's.  Tolerances: solutions to 1e-10 in the
residual carry errors of that order (end-loaded bars): 1e-9; the iteration
counts may differ by the rounding of the FP32 V-cycles, in the last steps: 3."""
import numpy as np
import pytest

from asend3d_gb300 import _lib
from asend3d_gb300.mesh import block_hex8
from asend3d_gb300.solver import GpuSolver, Problem, combine

pytestmark = pytest.mark.gpu

KW = dict(method=_lib.METHOD_SPLIT, precond=_lib.PC_MG, rel_tol=1e-10, max_iter=500)


def bar(dims, elem_type=8, seed=1, coupled=False):
    nx, ny, nz = dims
    rng = np.random.default_rng(seed)
    m = block_hex8(nx, ny, nz, 0.1 * nx, 0.07 * ny, 0.08 * nz)
    m.elem_type = elem_type
    p = Problem(m, 70e9 * np.exp(0.3 * rng.standard_normal(m.n_elems)), np.full(m.n_elems, 0.3))
    p.add_node_set("xMin", m.nodes_in_range(xr=(-1e-9, 1e-9)))
    p.fix_displacement("xMin")
    p.add_node_set("a", [int(m.node_id(nx, 0, 0))])
    p.add_node_set("b", [int(m.node_id(nx, 0, 1))])
    if coupled:
        p.constraints.append(([("a", 1, 1e-9), ("b", 1, -1e-9)], 0.0))
    end = m.nodes_in_range(xr=(0.1 * nx - 1e-9, 1e9))
    p.add_node_set("end", end)
    p.add_nodal_force("end", [300.0 / len(end), 0.0, -1000.0 / len(end)])
    return p


def matrix_free(g):
    m = g.p.mesh
    return g.time_mg_kernel(0, _lib.METHOD_SPLIT, 1)[1] == 8.0 * m.n_elems + 32.0 * m.n_nodes + 24.0 * m.n_nodes


def compare(make, expect=True):
    u, its = [], []
    for coupled in (False, True):
        p, inst, blocks = make(coupled)
        g = GpuSolver(p, instances=inst, blocks=blocks)
        g.assemble(48)
        for variant in ([_lib.PRODUCT_DEFAULT, _lib.PRODUCT_REGISTERS] if not coupled else [_lib.PRODUCT_DEFAULT]):
            g.set_product_variant(variant)
            x, rc, st = g.static_solve(**KW)
            assert rc == 0
            u.append(x[0])
            its.append(st["iterations"])
        g.set_product_variant(_lib.PRODUCT_DEFAULT)
        assert matrix_free(g) == (expect and not coupled)
        g.close()
    for k in (1, 2):
        assert np.linalg.norm(u[k] - u[0]) <= 1e-9 * np.linalg.norm(u[0])
        assert abs(its[k] - its[0]) <= 3


@pytest.mark.parametrize("dims,elem_type", [((9, 3, 3), 8), ((13, 4, 5), 81), ((30, 21, 19), 8), ((5, 40, 33), 81),
                                            ((3, 7, 190), 8), ((60, 5, 6), 8)])
def test_single_block(gpu_lib, dims, elem_type):
    compare(lambda coupled: (bar(dims, elem_type, coupled=coupled), None, None))


def test_long_rows_take_the_assembled_products(gpu_lib):
    compare(lambda coupled: (bar((3, 6, 191), coupled=coupled), None, None), expect=False)


def test_stack(gpu_lib):
    dims = [(20, 4, 4), (41, 9, 7), (8, 3, 5), (63, 12, 13)]

    def make(coupled):
        p, node_ptr, _ = combine([bar(d, seed=k, coupled=coupled) for k, d in enumerate(dims)])
        return p, node_ptr, dims

    compare(make)
