"""Captured iterations of a batch (m2d_ctx_set_graph on its instances) are
launched in pieces, the host reading each p' cycle's verdict.  Whatever the
number of passes and cycles, the iterates, the reports and the launch counts
are those of a lone context, and an instance may change between the batch and
its own calls."""
import numpy as np
import pytest

from mach2d_b200 import M2DError
from mach2d_b200.simplec import Batch, Simplec, euler_cosine_case, n01_case

pytestmark = pytest.mark.gpu
FIELDS = ("u", "v", "p", "T", "ro")


# one cycle per pass; a cap that is reached; the tolerance's own exit
@pytest.mark.parametrize("itmmax,itpmax,tolm", [(1, 1, 1e-2), (1, 3, 1e-30), (2, 20, 1e-2), (3, 2, 1e-30)])
def test_pieces_equal_the_host_loop(itmmax, itpmax, tolm):
    kw = dict(itmmax=itmmax, itpmax=itpmax, tolm=tolm)
    cases = [n01_case(**kw), euler_cosine_case(64, 32, **kw), euler_cosine_case(37, 11, **kw)]
    b = Batch(cases, workers=2)
    for s in b.instances:
        s.set_graph(True)
    b.iterate(5)
    b.instances[1].iterate()          # its own one-graph iteration in between
    b.instances[1].run(2)
    reps = b.iterate(4)
    for k, c in enumerate(cases):
        solo, graph = Simplec(c), Simplec(c)
        graph.set_graph(True)
        n = 12 if k == 1 else 9
        for _ in range(n):
            r = solo.iterate()
            graph.iterate()
        assert (reps[k].it, reps[k].itp_used, reps[k].norm, reps[k].rmass) == (n, r.itp_used, r.norm, r.rmass)
        assert b.instances[k].scalar("launches") == graph.scalar("launches")
        for f in FIELDS:
            assert np.array_equal(b.instances[k].field(f), solo.field(f)), (k, f)
        solo.close()
        graph.close()
    b.close()


def test_a_failed_instance_stops_and_the_others_go_on():
    b = Batch([n01_case() for _ in range(3)], workers=1)
    for s in b.instances:
        s.set_graph(True)
    b.iterate(1)
    g = b.instances[1]
    u = g.field("u")
    u[g.nx * 5 + 7] = np.nan
    g.set_field("u", u)
    with pytest.raises(M2DError) as e:
        b.iterate(3)
    assert e.value.code == 3 and "instance 1" in str(e.value)
    assert [s.scalar("it") for s in b.instances] == [4, 2, 4]
    b.close()
