"""The DST-I in block fixed point (csrc/fixed.cuh) against extended-precision sine matrices, over line
lengths that reach every radix, and its behaviour at the ends of the exponent range."""
import numpy as np
import pytest

from helpers import SMALL
from ib_parallel_gb300 import ibgpu as G

pytestmark = pytest.mark.gpu


def _sines(M):
    j = np.arange(1, M, dtype=np.int64)
    a = np.longdouble("3.14159265358979323846264338327950288")
    return 2 * np.sin(a * ((j[:, None] * j[None, :]) % (2 * M)).astype(np.longdouble) / M)


def _sim(m, n):
    return G.Simulation(G.Params(**dict(SMALL, m=m, n=n, mgridlev=1)), [])


def _rows(kind, n, m, rng):
    x = rng.standard_normal((n - 1, m - 1))
    if kind == "smooth":
        s = np.arange(1, m) / m
        x = np.exp(-((s[None, :] - rng.uniform(0.2, 0.8, (n - 1, 1))) / 0.05) ** 2)
    elif kind == "spikes":
        x *= rng.random(x.shape) < 0.01
        x[:, 0] += 1.0
    elif kind == "ranges":
        x *= 10.0 ** rng.uniform(-12.0, 0.0, x.shape)
    return x


# half lines of 4, 6, 10, 16, 18, 50, 200, 400, 768 and 1000 points: every radix first and last, lines
# shorter and longer than a warp and than the CTA.  Tolerance: an odd output is a sum of up to M/2
# increments, each within 2^-53 of the line's rms; the two passes add, and a factor 2 is left.
@pytest.mark.parametrize("mn", [(8, 12), (12, 8), (20, 36), (32, 64), (36, 20), (100, 48), (400, 200), (800, 60),
                                (1536, 40), (2000, 24)])
@pytest.mark.parametrize("kind", ["noise", "smooth", "spikes", "ranges"])
def test_dst_against_extended_precision(mn, kind):
    m, n = mn
    x = _rows(kind, n, m, np.random.default_rng(m + n))
    g = _sim(m, n)
    y = g.dst(x)
    g.close()
    exact = _sines(n) @ x.astype(np.longdouble) @ _sines(m)
    err = float(np.linalg.norm((y - exact).astype(np.float64)) / np.linalg.norm(exact.astype(np.float64)))
    assert err < 2 * 2.0 ** -53 * (np.sqrt(m / 2) + np.sqrt(n / 2))


def test_dst_exponents():
    """A power of two factors out exactly; zeros stay zeros; results past the range become infinite or
    subnormal; a sample that is not finite makes its line NaN and stops nothing."""
    g = _sim(64, 32)
    x = np.random.default_rng(5).standard_normal((31, 63))
    y = g.dst(x)
    for k in (-900, -300, 300, 900):
        assert np.array_equal(g.dst(x * 2.0 ** k), y * 2.0 ** k)
    assert not g.dst(np.zeros_like(x)).any()
    small = g.dst(x * 2.0 ** -1060)
    assert np.isfinite(small).all() and np.abs(small - y * 2.0 ** -1060).max() <= 64 * 5e-324 * np.abs(y).max()
    assert np.isinf(g.dst(np.full_like(x, 1e308))).any()
    for bad in (np.nan, np.inf):
        z = x.copy()
        z[3, 7] = bad
        assert np.isnan(g.dst(z)).all()   # its row, then through the columns every value
    assert np.array_equal(g.dst(x), y)
    g.close()
