"""Line batches at the edges of the launcher's rule: one or four lines per CTA,
P and Q in shared or global memory, one thread per line.  Every line's bits are
those of the recurrence in plain FP64 (numpy, all lines at once)."""
import numpy as np
import pytest

from mach2d_b200.solvers import tdma_lines

pytestmark = pytest.mark.gpu


def _recurrence(aw, ap, ae, d):
    P, Q, x = np.zeros_like(ap), np.zeros_like(ap), np.zeros_like(ap)
    n = ap.shape[1]
    P[:, 0], Q[:, 0] = -ae[:, 0] / ap[:, 0], d[:, 0] / ap[:, 0]
    for i in range(1, n):
        den = ap[:, i] + aw[:, i] * P[:, i - 1]
        P[:, i] = -ae[:, i] / den
        Q[:, i] = (d[:, i] - aw[:, i] * Q[:, i - 1]) / den
    x[:, n - 1] = Q[:, n - 1]
    for i in range(n - 2, -1, -1):
        x[:, i] = P[:, i] * x[:, i + 1] + Q[:, i]
    return x


@pytest.mark.parametrize("n,nlines", [
    (300, 999), (300, 1000), (65, 1003), (768, 1001), (769, 1001),      # one line per CTA, four
    (1199, 2401), (1200, 2399), (1200, 2402),                           # four, P and Q in global memory
    (16, 4095), (16, 4096), (17, 4096), (1, 5000),                      # one thread per line
    (63, 19999), (63, 20000), (64, 20001)])
def test_every_line_bitwise(n, nlines):
    rng = np.random.default_rng(n + nlines)
    aw, ae = -rng.random((nlines, n)), -rng.random((nlines, n))
    aw[:, 0] = 0.0
    ae[:, -1] = 0.0
    ap = 1.05 * (np.abs(aw) + np.abs(ae)) + 1e-3
    d = rng.standard_normal((nlines, n))
    d[rng.random((nlines, n)) < 0.2] *= 0.0                             # zeros of both signs
    x, xr = tdma_lines(aw, ap, ae, d), _recurrence(aw, ap, ae, d)
    assert np.array_equal(x, xr) and np.array_equal(np.signbit(x), np.signbit(xr))
