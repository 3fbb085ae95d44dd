"""Host threads of a batch launch the same kernels at different grid sizes at
the same time: a launch's shared-memory limit must not be another thread's."""
import numpy as np
import pytest

from mach2d_b200.simplec import Batch, Simplec, euler_cosine_case

pytestmark = pytest.mark.gpu


# line TDMA and the one-CTA MSI kernel take shared memory by the grid's size
@pytest.mark.parametrize("solver,schedule", [(1, 0), (0, 3)])
def test_threads_launch_uneven_grids(solver, schedule):
    sizes = [(20, 9), (199, 150), (64, 33), (400, 260), (36, 130), (150, 64)]
    cases = [euler_cosine_case(nx, ny, solver=solver) for nx, ny in sizes]
    b = Batch(cases, workers=6)
    for s in b.instances:
        s.set_msi_schedule(schedule)
    reps = b.iterate(20)
    for k in (0, 2, 3):
        solo = Simplec(cases[k])
        for _ in range(20):
            r = solo.iterate()
        assert reps[k].norm == r.norm
        for f in ("u", "p"):
            assert np.array_equal(b.instances[k].field(f), solo.field(f)), (k, f)
        solo.close()
    b.close()
