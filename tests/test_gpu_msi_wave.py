"""The cluster MSI kernel at the edges of its row groups (32 rows), batches
(8, 16 or 32 lines) and cluster shapes (one group per CTA, two from 513 rows
on): FP64 bitwise against the oracle over several iterations, the repeat of
a forward sweep whose operands leave the checked range, and the FP32-factor
solve to a tolerance it must reach."""
import numpy as np
import pytest

from _oracle import call as orc
from _systems import dirichlet_system, random_dominant_planes
from mach2d_b200.solvers import ClassSolverMSI5d, ClassSolverMSI9d, ClassSolverMSIMixed5d, ClassSolverMSIMixed9d

pytestmark = pytest.mark.gpu

SHAPES = [(4, 4), (4, 33), (5, 65), (17, 32), (18, 64), (19, 31), (34, 97), (66, 66), (67, 34), (98, 128),
          (21, 512), (24, 513), (9, 545), (13, 1024)]


@pytest.mark.parametrize("nd", [9, 5])
@pytest.mark.parametrize("nx,ny", SHAPES)
def test_fp64_bitwise(nd, nx, ny):
    a, b = random_dominant_planes(nd, nx, ny, seed=nx + ny)
    x0 = np.random.default_rng(ny).standard_normal(nx * ny)
    xg, xo = x0.copy(), x0.copy()
    s = (ClassSolverMSI9d if nd == 9 else ClassSolverMSI5d)().init(nx, ny, 3, 1e-30)
    s.solve(a, b, xg)
    assert s.nit == orc(f"msi{nd}_solve", nx, ny, 3, 1e-30, a, b, xo)
    assert np.array_equal(xg, xo), np.max(np.abs(xg - xo))


@pytest.mark.parametrize("nd", [9, 5])
@pytest.mark.parametrize("nx,ny", [(30, 96), (37, 64), (12, 40)])
def test_scaled_equations(nd, nx, ny):
    # reciprocal pivots of 2^200: a line that is not the group's must not reach
    # the backward sweep through its last, partly filled batch
    a, b = random_dominant_planes(nd, nx, ny, seed=6)
    a, b = a * 2.0 ** -200, b * 2.0 ** -200
    xg, xo = np.zeros(nx * ny), np.zeros(nx * ny)
    s = (ClassSolverMSI9d if nd == 9 else ClassSolverMSI5d)().init(nx, ny, 2, 1e-30)
    s.solve(a, b, xg)
    assert s.nit == orc(f"msi{nd}_solve", nx, ny, 2, 1e-30, a, b, xo)
    assert np.array_equal(xg, xo), np.max(np.abs(xg - xo))


@pytest.mark.parametrize("nd", [9, 5])
@pytest.mark.parametrize("e", [-600, 600])
def test_forward_operands_out_of_range(nd, e):
    # the factors do not see the right-hand side; its sweep must go back to '/'
    nx, ny = 45, 70
    a, b = random_dominant_planes(nd, nx, ny, seed=5)
    b = b * 2.0 ** e
    xg, xo = np.zeros(nx * ny), np.zeros(nx * ny)
    s = (ClassSolverMSI9d if nd == 9 else ClassSolverMSI5d)().init(nx, ny, 3, 1e-30)
    s.solve(a, b, xg)
    assert s.nit == orc(f"msi{nd}_solve", nx, ny, 3, 1e-30, a, b, xo)
    assert np.array_equal(xg, xo), np.max(np.abs(xg - xo))


@pytest.mark.parametrize("nd", [9, 5])
@pytest.mark.parametrize("scale", [1.0, 1e-6])
@pytest.mark.parametrize("nx,ny", [(12, 10), (40, 33), (66, 66), (30, 96), (24, 513)])
def test_fp32_factors_reach_the_tolerance(nd, nx, ny, scale):
    # |r| < tol |r0| and a diagonal dominance of 1.05 bound the error by
    # tol |b| / (0.05 min aP) up to norms: compared with the FP64 solution at
    # a tolerance 1e3 above the residuals'
    a, b = dirichlet_system(nd, nx, ny, seed=3)
    a *= scale
    xg, xo = np.zeros(nx * ny), np.zeros(nx * ny)
    s = (ClassSolverMSIMixed9d if nd == 9 else ClassSolverMSIMixed5d)().init(nx, ny, 400, 1e-11)
    s.solve(a, b, xg)
    orc(f"msi{nd}_solve", nx, ny, 400, 1e-11, a, b, xo)
    assert s.nit < 400
    assert np.linalg.norm(xg - xo) <= 1e-8 * np.linalg.norm(xo)


@pytest.mark.parametrize("nd", [9, 5])
def test_fill_in_that_decays_below_the_normal_range(nd):
    # rows whose factors decay geometrically along x, through 2^-900 and the
    # subnormals; x agrees with the oracle to one subnormal unit per term
    nx, ny = 700, 40
    a, b = random_dominant_planes(nd, nx, ny, seed=8)
    a = a.reshape(nd, ny, nx)
    off = 4 if nd == 9 else 2
    for k in range(nd):
        if k != off:
            a[k] *= 2.0 ** -4
    b = np.where(np.arange(nx * ny) % nx < 3, b, 0.0)
    a = a.reshape(-1).copy()
    xg, xo = np.zeros(nx * ny), np.zeros(nx * ny)
    s = (ClassSolverMSI9d if nd == 9 else ClassSolverMSI5d)().init(nx, ny, 2, 1e-30)
    s.solve(a, b, xg)
    assert s.nit == orc(f"msi{nd}_solve", nx, ny, 2, 1e-30, a, b, xo)
    assert np.max(np.abs(xg - xo)) <= 64 * 2.0 ** -1074
