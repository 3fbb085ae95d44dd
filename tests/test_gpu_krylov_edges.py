"""m2d_fgmres_solve where its multi-dot's split can go wrong: restarts around
the four rows a block takes, up to the largest; fewer cells than slices, rows
of one block and one more.  The residual the solver reports is its own dot of
b - A x: it must meet the tolerance and be numpy's."""
import numpy as np
import pytest

from _systems import dirichlet_system
from mach2d_b200.solvers import fgmres
from test_gpu_krylov import _residual

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(4, 4), (5, 61), (128, 4), (129, 33), (257, 130)])
@pytest.mark.parametrize("nd,restart", [(9, 3), (9, 5), (5, 4), (5, 32)])
def test_fgmres_at_the_edges(nd, restart, nx, ny):
    import torch
    tol = 1e-10
    a, b = dirichlet_system(nd, nx, ny, seed=7 * nx + ny + nd)
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    runs = []
    for _ in range(2):
        x = torch.zeros(nx * ny, dtype=torch.float64, device="cuda")
        rep = fgmres(nd, nx, ny, da, db, x, tol, restart=restart)
        assert rep.converged == 1
        runs.append(x.cpu().numpy())
    assert np.array_equal(runs[0], runs[1])
    got = _residual(nd, nx, ny, a, b, runs[0])
    assert got <= tol * 1.001 and abs(rep.rel_residual - got) <= 1e-13
