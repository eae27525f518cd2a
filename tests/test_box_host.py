"""The matrix-free products of k_box.cu on the CPU, from their own source
(box_host.cpp): the same results in whatever order the threads of a CTA run
between barriers, and every row against the element-by-element product in
extended precision.

Tolerances.  With u the rounding unit of the arithmetic (FP32 2^-24, pairs
2^-47: TwoSum with the errors carried) a row's value passes through at most 30
roundings one after the other (two sums a direction in and out of the sign
patterns, a product of three with its scaling, eight contributions), each of a
value bounded by the sum of |E K^| |x| over the node's elements with K^ taken
through the patterns (64 |B| entries: at most the largest row sum of |K^| times
|x|'s largest): |y - ref| <= 30 u (sum_e E_e) max_row(|K^|) max|x|."""
import ctypes as C
import re
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "asend3d_gb300" / "csrc"
CORNER = np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0], [0, 0, 1], [1, 0, 1], [1, 1, 1], [0, 1, 1]])
PRODUCT, RESID, POST, POWER = range(4)


def between(text, start, stop):
    a = text.index(start)
    return text[a:text.index(stop, a)]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    box, pcg = (CSRC / "k_box.cu").read_text(), (CSRC / "pcg_common.cuh").read_text()
    code = between(pcg, "__device__ __forceinline__ void split_term", "// alpha = r.z")
    code += between(box, "struct BoxItem {", "struct BoxPlan {")
    code += between(box, "constexpr int kBoxThreads", "BoxArgs args_of")
    code = re.sub(r"extern __shared__.*;", "", code)  # box_host.cpp's buffer
    code = code.replace("__shared__", "static")
    tmp = tmp_path_factory.mktemp("box")
    (tmp / "box_kernels.inc").write_text(code)
    so = tmp / "libbox.so"
    subprocess.run([shutil.which("g++") or "c++", "-O2", "-std=c++17", "-ffp-contract=off", "-w", "-fPIC", "-shared",
                    f"-I{tmp}", str(ROOT / "tests" / "box_host.cpp"), "-o", str(so)], check=True)
    return C.CDLL(str(so))


def box_stiffness(h, nu=0.3):
    """K^ of a box hex8 at unit modulus (2 x 2 x 2 Gauss points)."""
    lam, mu = nu / ((1 + nu) * (1 - 2 * nu)), 0.5 / (1 + nu)
    D = np.diag([2 * mu] * 3 + [mu] * 3)
    D[:3, :3] += lam
    K = np.zeros((24, 24))
    sg = 2.0 * CORNER - 1.0
    g = 1 / np.sqrt(3)
    for q in range(8):
        s = g * sg[q]
        f = 1 + sg * s
        dN = np.stack([0.125 * sg[:, 0] * f[:, 1] * f[:, 2], 0.125 * sg[:, 1] * f[:, 0] * f[:, 2],
                       0.125 * sg[:, 2] * f[:, 0] * f[:, 1]], 1) * 2 / np.asarray(h)
        Bm = np.zeros((6, 24))
        for a in range(8):
            x, y, z = dN[a]
            Bm[:, 3 * a:3 * a + 3] = [[x, 0, 0], [0, y, 0], [0, 0, z], [y, x, 0], [0, z, y], [z, 0, x]]
        K += Bm.T @ D @ Bm * np.prod(h) / 8
    return K


def pair(v):
    hi = v.astype(np.float32)
    return np.stack([hi, (v - hi).astype(np.float32)], -1)


def value(p):
    return p[..., 0].astype(np.longdouble) + p[..., 1].astype(np.longdouble)


class Case:
    def __init__(self, dims, pad=0, seed=0):
        rng = np.random.default_rng(seed)
        blocks, node0, el0, conn = [], 0, 0, []
        for nx, ny, nz in dims:
            blocks.append((nx, ny, nz, node0, el0))
            i, j, k = (a.ravel() for a in np.meshgrid(range(nx), range(ny), range(nz), indexing="ij"))
            conn.append(np.stack([node0 + ((i + a) * (ny + 1) + j + b) * (nz + 1) + k + c for a, b, c in CORNER], 1))
            node0 += (nx + 1) * (ny + 1) * (nz + 1) + pad
            el0 += nx * ny * nz
        self.blocks, self.n, self.conn = np.array(blocks, np.int32), node0, np.concatenate(conn)
        self.K = box_stiffness((0.1, 0.07, 0.08))
        self.E = pair(np.exp(0.3 * rng.standard_normal(el0)))
        self.pen = np.zeros((3 * node0, 2), np.float32)
        used = np.unique(self.conn)
        at = rng.choice(3 * used.size, used.size // 3, replace=False)
        self.pen[3 * used[at // 3] + at % 3] = pair(1e3 * (1 + rng.random(at.size)))
        self.x = pair(rng.standard_normal((node0, 3)))
        self.b = rng.standard_normal((node0, 3)).astype(np.float32)
        self.binv = rng.standard_normal((node0, 3, 3)).astype(np.float32)
        self.unit = np.setdiff1d(np.arange(node0), used)  # padding: unit rows

    def reference(self, x):
        """A x and, per node, the scale of its rounding errors."""
        E, K = value(self.E), self.K.astype(np.longdouble)
        ye = E[:, None] * (x[self.conn].reshape(-1, 24) @ K.T)
        y = np.zeros((self.n, 3), np.longdouble)
        scale = np.zeros(self.n)
        for a in range(8):
            np.add.at(y, self.conn[:, a], ye[:, 3 * a:3 * a + 3])
            np.add.at(scale, self.conn[:, a], self.E[:, 0])
        pen = value(self.pen).reshape(-1, 3)
        y += pen * x
        y[self.unit] = x[self.unit]
        scale = scale * np.abs(self.K).sum(1).max() + pen.max(1).astype(float)
        scale[self.unit] = 1.0
        return y, scale[:, None] * float(np.abs(x).max())

    def run(self, lib, kind, sms, down=False):
        x = np.zeros((self.n, 2, 4) if kind == PRODUCT else (self.n, 1, 4), np.float32)
        x[:, 0, :3] = self.x[..., 0]
        if kind == PRODUCT:
            x[:, 1, :3] = self.x[..., 1]
        out = np.full((self.n, 3, 2) if kind == PRODUCT else (self.n, 3 if kind == RESID else 4), np.nan, np.float32)
        part, shape = np.full(100000, np.nan), np.zeros(2, np.int32)
        p = lambda a: a.ctypes.data_as(C.c_void_p)
        n = lib.box_launch(kind, len(self.blocks), p(self.blocks), self.n, sms, p(self.K), p(self.E), p(self.pen), p(x),
                           p(self.b), p(self.binv), int(down), p(out), p(part), p(shape))
        assert n <= part.size
        return out, part[:1 if kind == PRODUCT else n if kind == POWER else 0], shape


# planes a CTA: several and one; a plane in one CTA and in several; a stack with padding
CASES = [(((9, 3, 3),), 0, 1), (((9, 3, 3),), 0, 152), (((13, 4, 5),), 0, 2), (((5, 40, 33),), 0, 4),
         (((3, 2, 190),), 0, 1), (((1, 1, 1),), 0, 1), (((6, 4, 4), (11, 9, 7), (8, 3, 5)), 13, 2)]


@pytest.mark.parametrize("dims,pad,sms", CASES)
@pytest.mark.parametrize("kind", [PRODUCT, RESID, POST, POWER])
def test_thread_order_does_not_matter(lib, kind, dims, pad, sms):
    c = Case(dims, pad)
    up, down = c.run(lib, kind, sms), c.run(lib, kind, sms, down=True)
    assert np.array_equal(up[0], down[0])
    if sms == 1 and c.n > 8:
        assert up[2][1] > 1  # planes a CTA


@pytest.mark.parametrize("dims,pad,sms", CASES)
def test_rows(lib, dims, pad, sms):
    c = Case(dims, pad)
    x = value(c.x)
    y, scale = c.reference(x)
    out, dot, _ = c.run(lib, PRODUCT, sms)
    assert (np.abs(value(out) - y) <= 30 * 2.0**-47 * scale).all()
    assert abs(dot[0] - (x * y).sum()) <= 60 * 2.0**-47 * float((np.abs(x) * scale).sum())
    x32 = c.x[..., 0].astype(np.longdouble)
    y, scale = c.reference(x32)
    tol = 30 * 2.0**-24 * scale
    assert (np.abs(c.run(lib, RESID, sms)[0] - (c.b - y)) <= tol + 2.0**-23 * np.abs(c.b)).all()
    post = x32 + np.einsum("nij,nj->ni", c.binv.astype(np.longdouble), c.b - y)
    grow = np.abs(c.binv).sum(2)
    size = np.abs(c.b).max() + scale
    assert (np.abs(c.run(lib, POST, sms)[0][:, :3] - post) <= grow * (tol + 2.0**-22 * size) + 2.0**-23 * 5).all()


@pytest.mark.parametrize("dims,pad,sms", CASES)
def test_power_step_sums_in_64_bits(lib, dims, pad, sms):
    """The CTAs' sums of the new vector's squares, positive terms: each addition
    and product rounds by 2^-53."""
    c = Case(dims, pad)
    y, part, _ = c.run(lib, POWER, sms)
    exact = (y[:, :3].astype(np.longdouble) ** 2).sum()
    assert abs(part.sum(dtype=np.longdouble) - exact) <= 2 * y.size * 2.0**-53 * exact
