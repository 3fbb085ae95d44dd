"""The line TDMA kernel at the edges of its chunks (64 elements) and of a
CTA's lines (one x line, four y lines), with lines too long for shared memory,
and with quotients that need IEEE division: bitwise against the oracle."""
import numpy as np
import pytest

from _oracle import call as orc
from _systems import random_dominant_planes, tdma_lines_system
from mach2d_b200.solvers import ClassSolverTDMA5d, ClassSolverTDMA9d, tdma_lines

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nd", [9, 5])
@pytest.mark.parametrize("nx,ny", [(4, 4), (63, 5), (64, 6), (65, 7), (5, 64), (6, 129), (130, 9), (4000, 5), (5, 4000)])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -1010])
def test_tdma_bitwise(nd, nx, ny, scale):
    a, b = random_dominant_planes(nd, nx, ny, seed=nx + ny)
    a, b = a * scale, b * scale      # 2^-1010: remainders underflow, '/' must take over
    x0 = np.random.default_rng(nx).standard_normal(nx * ny)
    xg, xo = x0.copy(), x0.copy()
    s = (ClassSolverTDMA9d if nd == 9 else ClassSolverTDMA5d)().init(nx, ny, 2)
    s.solve(a, b, xg)
    orc(f"tdma2d{nd}", nx, ny, 2, a, b, xo)
    assert np.array_equal(xg, xo), np.max(np.abs(xg - xo))


@pytest.mark.parametrize("n,nlines", [(1, 3), (2, 1), (64, 5), (65, 2), (16000, 3)])
def test_lines_bitwise(n, nlines):
    aw, ap, ae, d = tdma_lines_system(n=n, nlines=nlines, seed=n)
    x = tdma_lines(aw, ap, ae, d)
    for k in range(nlines):
        xo = np.zeros(n)
        orc("tdma_line", n, aw[k].copy(), ap[k].copy(), ae[k].copy(), d[k].copy(), xo)
        assert np.array_equal(x[k], xo)
