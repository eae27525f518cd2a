"""Newmark runs in the one-launch PCG end a launch after some thousand iterations:
the steps go on where the last launch stopped, and another context's solves come
in between.  Histories of the two routes, each step solved to 1e-12: 1e-8 (the
increments' errors, 1e-12 times a time operator's condition below 1e3, over the
steps of a run)."""
import threading
import time

import numpy as np
import pytest

from asend3d_gb300 import _lib
from asend3d_gb300.mesh import block_hex8
from asend3d_gb300.solver import GpuSolver, Problem

pytestmark = pytest.mark.gpu

KW = dict(precond=_lib.PC_JACOBI, rel_tol=1e-12)


def solver(dims, **kw):
    nx, ny, nz = dims
    rng = np.random.default_rng(4)
    m = block_hex8(nx, ny, nz, 0.1 * nx, 0.1 * ny, 0.1 * nz)
    p = Problem(m, 70e9 * np.exp(0.3 * rng.standard_normal(m.n_elems)), np.full(m.n_elems, 0.3),
                np.full(m.n_elems, 2700.0))
    p.add_node_set("xMin", m.nodes_in_range(xr=(-1e-9, 1e-9)))
    p.fix_displacement("xMin")
    p.add_load_vector(1000.0 * rng.standard_normal(m.n_dof))
    g = GpuSolver(p)
    g.assemble(64, **kw)
    return g


@pytest.mark.parametrize("warm_start", [0, 2])
@pytest.mark.parametrize("loaded", [True, False])
def test_several_launches(gpu_lib, warm_start, loaded):
    steps = 300 if loaded else 10000  # without a load a step has no iterations
    amp = np.sin(0.1 * np.arange(steps)) if loaded else np.zeros(steps)
    runs = []
    for method in (_lib.METHOD_FP64, _lib.METHOD_SPLIT) if loaded else (_lib.METHOD_FP64,):
        g = solver((16, 4, 4), dynamic=True, dt=2e-5)
        before = g.kernel_launches
        hist, u, rc, st = g.newmark(amp, probe_dof=g.n_dof - 1, method=method, warm_start=warm_start, **KW)
        assert rc == 0
        runs.append((hist, u, g.kernel_launches - before, st["iterations"]))
        g.close()
    hist, u, launches, its = runs[0]
    if not loaded:
        assert its == 0 and not hist.any() and not u.any()
        assert 3 <= launches <= 16
        return
    assert its > 2048 and 3 <= launches <= its // 1024 + 5
    assert np.abs(hist - runs[1][0]).max() <= 1e-8 * np.abs(hist).max()
    assert np.linalg.norm(u - runs[1][1]) <= 1e-8 * np.linalg.norm(u)


def test_other_contexts_come_in_between(gpu_lib):
    """Solves of a few ms beside a run of seconds end before it does."""
    a, b = solver((20, 4, 4), dynamic=True, dt=2e-5), solver((57, 13, 11))
    kw = dict(method=_lib.METHOD_FP64, precond=_lib.PC_JACOBI)
    b.static_solve(rel_tol=1e-3, **kw)
    t = time.perf_counter()
    a.newmark(np.ones(200), rel_tol=1e-8, **kw)
    steps = int(200 * 2.0 / (time.perf_counter() - t))
    rc = []
    run = threading.Thread(target=lambda: rc.append(a.newmark(np.ones(steps), rel_tol=1e-8, **kw)[2]))
    run.start()
    time.sleep(0.2)
    for _ in range(3):
        assert b.static_solve(rel_tol=1e-3, **kw)[1] == 0
    assert run.is_alive()
    run.join()
    assert rc == [0]
    a.close()
    b.close()
