"""FP64 quotients at the ends of the range: the solvers divide with refined
reciprocal approximations and must notice every quotient that is not IEEE
division's."""
import ctypes

import numpy as np
import pytest

from _oracle import call as orc
from _systems import random_dominant_planes, tdma_lines_system
from mach2d_b200._lib import lib
from mach2d_b200.solvers import (ClassSolverMSI5d, ClassSolverMSI9d, ClassSolverTDMA5d, ClassSolverTDMA9d,
                                 tdma_lines)

pytestmark = pytest.mark.gpu


def _huge_diagonals(nd, nx, ny, seed, e=1022):
    """A fifth of the equations with a diagonal in [2^e, 2^(e+1)); for e = 1022
    its reciprocal is subnormal.  Every quotient of theirs is a normal number."""
    a, b = random_dominant_planes(nd, nx, ny, seed=seed)
    rng = np.random.default_rng(seed + 1)
    rows = rng.random(nx * ny) < 0.2
    a = a.reshape(nd, -1)
    a[:, rows] *= 2.0 ** 150
    a[4 if nd == 9 else 2, rows] = rng.uniform(1.0, 2.0, rows.sum()) * 2.0 ** e
    b[rows] *= 2.0 ** 500
    return a.reshape(-1).copy(), b


@pytest.mark.parametrize("nd", [9, 5])
@pytest.mark.parametrize("nx,ny", [(20, 35), (45, 70)])
def test_msi_with_huge_diagonals(nd, nx, ny):
    a, b = _huge_diagonals(nd, nx, ny, seed=nx)
    xg, xo = np.zeros(nx * ny), np.zeros(nx * ny)
    s = (ClassSolverMSI9d if nd == 9 else ClassSolverMSI5d)().init(nx, ny, 3, 1e-30)
    s.solve(a, b, xg)
    assert s.nit == orc(f"msi{nd}_solve", nx, ny, 3, 1e-30, a, b, xo)
    assert np.array_equal(xg, xo), np.max(np.abs(xg - xo))


@pytest.mark.parametrize("nd", [9, 5])
@pytest.mark.parametrize("e", [890, 894, 896, 930, 1000])
def test_msi_where_a_scaled_remainder_overflows(nd, e):
    a, b = _huge_diagonals(nd, 45, 70, seed=e, e=e)
    xg, xo = np.zeros(45 * 70), np.zeros(45 * 70)
    s = (ClassSolverMSI9d if nd == 9 else ClassSolverMSI5d)().init(45, 70, 2, 1e-30)
    s.solve(a, b, xg)
    assert s.nit == orc(f"msi{nd}_solve", 45, 70, 2, 1e-30, a, b, xo)
    assert np.array_equal(xg, xo), np.max(np.abs(xg - xo))


@pytest.mark.parametrize("nd", [9, 5])
@pytest.mark.parametrize("nx,ny", [(20, 35), (70, 45)])
def test_tdma_with_huge_diagonals(nd, nx, ny):
    a, b = _huge_diagonals(nd, nx, ny, seed=ny)
    xg, xo = np.zeros(nx * ny), np.zeros(nx * ny)
    (ClassSolverTDMA9d if nd == 9 else ClassSolverTDMA5d)().init(nx, ny, 2).solve(a, b, xg)
    orc(f"tdma2d{nd}", nx, ny, 2, a, b, xo)
    assert np.array_equal(xg, xo), np.max(np.abs(xg - xo))


@pytest.mark.parametrize("n", [3, 200])
def test_lines_with_huge_diagonals(n):
    aw, ap, ae, d = tdma_lines_system(n=n, nlines=4, seed=n)
    ap[:, 1::3] = np.random.default_rng(n).uniform(1.0, 2.0, ap[:, 1::3].shape) * 2.0 ** 1022
    aw[:, 1::3] *= 2.0 ** 150
    ae[:, 1::3] *= 2.0 ** 150
    d[:, 1::3] *= 2.0 ** 500
    x = tdma_lines(aw, ap, ae, d)
    for k in range(4):
        xo = np.zeros(n)
        orc("tdma_line", n, aw[k].copy(), ap[k].copy(), ae[k].copy(), d[k].copy(), xo)
        assert np.array_equal(x[k], xo)


def _wall(nd, nx, ny, lo, hi, seed):
    """Rows coupled to the west only, but for a north coupling in the first
    cell of each: the fill-in u of the factorisation decays along x, through the
    subnormals.  The right-hand side is zero in every other row: there x is
    -u z of the row above, subnormals included."""
    rng = np.random.default_rng(seed)
    a = np.zeros((nd, ny, nx))
    w, p, n = (3, 4, 7) if nd == 9 else (1, 2, 4)
    a[w, :, 1:] = -rng.uniform(0.5, 1.0, (ny, nx - 1)) * 2.0 ** -4
    a[p] = rng.uniform(lo, hi, (ny, nx))
    a[n, :-1, 0] = -1.0
    b = np.where(np.arange(ny)[:, None] % 2 == 1, rng.standard_normal((ny, nx)), 0.0)
    return a.reshape(-1).copy(), b.reshape(-1).copy()


@pytest.mark.parametrize("nd", [9, 5])
@pytest.mark.parametrize("nx,ny,lo,hi", [(500, 20, 1.5, 1.9), (640, 40, 3.0, 4.0)])
def test_msi_fill_in_through_the_subnormals(nd, nx, ny, lo, hi):
    a, b = _wall(nd, nx, ny, lo, hi, seed=nx)
    xg, xo = np.zeros(nx * ny), np.zeros(nx * ny)
    s = (ClassSolverMSI9d if nd == 9 else ClassSolverMSI5d)().init(nx, ny, 1, 1e-30)
    s.solve(a, b, xg)
    orc(f"msi{nd}_solve", nx, ny, 1, 1e-30, a, b, xo)
    below = (np.abs(xo) < 2.0 ** -1022) & (xo != 0.0)
    assert below.any()
    assert np.array_equal(xg, xo), np.max(np.abs(xg - xo))


@pytest.mark.parametrize("nd", [9, 5])
def test_msi_fill_in_needs_no_repeat(nd):
    nx, ny = 640, 40
    a, b = _wall(nd, nx, ny, 1.5, 4.0, seed=1)
    L = lib()
    L.m2d_msi_lu_redo_count.restype = ctypes.c_longlong
    before = L.m2d_msi_lu_redo_count()
    (ClassSolverMSI9d if nd == 9 else ClassSolverMSI5d)().init(nx, ny, 1, 1e-30).solve(a, b, np.zeros(nx * ny))
    assert L.m2d_msi_lu_redo_count() == before


@pytest.mark.parametrize("nd", [9, 5])
def test_tdma_through_the_subnormals(nd):
    a, b = random_dominant_planes(nd, 700, 9, seed=8)
    a = a.reshape(nd, -1)
    for k in range(nd):
        if k != (4 if nd == 9 else 2):
            a[k] *= 2.0 ** -4
    b = np.where(np.arange(700 * 9) % 700 < 3, b, 0.0)
    xg, xo = np.zeros(700 * 9), np.zeros(700 * 9)
    (ClassSolverTDMA9d if nd == 9 else ClassSolverTDMA5d)().init(700, 9, 2).solve(a.reshape(-1), b, xg)
    orc(f"tdma2d{nd}", 700, 9, 2, a.reshape(-1).copy(), b, xo)
    assert ((np.abs(xo) < 2.0 ** -1022) & (xo != 0.0)).any()
    assert np.array_equal(xg, xo), np.max(np.abs(xg - xo))


@pytest.mark.parametrize("scale", [0.4, 1.0, 40.0])
def test_lines_through_the_subnormals(scale):
    n = 700
    aw, ap, ae, d = tdma_lines_system(n=n, nlines=6, seed=3)
    ap = scale * np.random.default_rng(5).uniform(1.0, 2.0, ap.shape)
    aw, ae = scale * aw * 2.0 ** -4, scale * ae * 2.0 ** -4
    d[:, 3:] = 0.0
    x = tdma_lines(aw, ap, ae, d)
    for k in range(6):
        xo = np.zeros(n)
        orc("tdma_line", n, aw[k].copy(), ap[k].copy(), ae[k].copy(), d[k].copy(), xo)
        assert ((np.abs(xo) < 2.0 ** -1022) & (xo != 0.0)).any()
        assert np.array_equal(x[k], xo)


def _same_bits(x, y):
    return np.array_equal(x, y) and np.array_equal(np.signbit(x), np.signbit(y))


@pytest.mark.parametrize("n", [1, 5, 130])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_lines_keep_the_sign_of_a_zero(n, sign):
    aw, ap, ae, d = tdma_lines_system(n=n, nlines=8, seed=n)
    rng = np.random.default_rng(n + 1)
    for v in (aw, ae, d):
        v[rng.random(v.shape) < 0.5] *= 0.0        # zeros of both signs
    d[:4] *= 0.0
    ap *= sign
    x = tdma_lines(aw, ap, ae, d)
    for k in range(8):
        xo = np.zeros(n)
        orc("tdma_line", n, aw[k].copy(), ap[k].copy(), ae[k].copy(), d[k].copy(), xo)
        assert _same_bits(x[k], xo)


@pytest.mark.parametrize("nd", [9, 5])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_tdma_keeps_the_sign_of_a_zero(nd, sign):
    nx, ny = 70, 30
    a, b = random_dominant_planes(nd, nx, ny, seed=11)
    rng = np.random.default_rng(12)
    a = sign * a.reshape(nd, -1)
    for k in range(nd):
        if k != (4 if nd == 9 else 2):
            a[k, rng.random(nx * ny) < 0.6] *= 0.0
    b[rng.random(nx * ny) < 0.8] *= 0.0
    x0 = np.where(rng.random(nx * ny) < 0.5, -0.0, 0.0)
    xg, xo = x0.copy(), x0.copy()
    (ClassSolverTDMA9d if nd == 9 else ClassSolverTDMA5d)().init(nx, ny, 1).solve(a.reshape(-1), b, xg)
    orc(f"tdma2d{nd}", nx, ny, 1, a.reshape(-1).copy(), b, xo)
    assert (xo == 0.0).any()
    assert _same_bits(xg, xo)
