"""The pressure's x transform (csrc/pressure.cu, the digit products) alone, against extended-precision sine
sums: half lines about a tile (32 terms), about a summation chunk (512) and about two chunks; its error
beside the FP64 product's; and the ends of the exponent range."""
import numpy as np
import pytest

from helpers import SMALL
from ib_parallel_gb300 import ibgpu as G

pytestmark = pytest.mark.gpu

LD = np.longdouble


def _sines(m):
    M = m + 1
    j = np.arange(1, M, dtype=np.int64)
    tab = 2 * np.sin(LD("3.14159265358979323846264338327950288") * np.arange(2 * M).astype(LD) / M)
    return tab[(j[:, None] * j[None, :]) % (2 * M)]


def _sim(m, n):
    return G.Simulation(G.Params(**dict(SMALL, m=m, n=n, mgridlev=1)), [])


def _rows(kind, n, m, rng):
    s = np.arange(1, m + 1)[None, :] / (m + 1)
    if kind == "smooth":
        return np.exp(-((s - rng.uniform(0.2, 0.8, (n, 1))) / 0.05) ** 2)
    x = rng.standard_normal((n, m))
    if kind == "decades":
        x *= 10.0 ** rng.uniform(-12.0, 0.0, x.shape)
    elif kind == "spike":
        x *= 1e-6
        x[np.arange(n), (np.arange(n) * m) // n] += 1.0
    return x


KINDS = ["noise", "smooth", "decades", "spike"]


# tolerance: the folded samples are multiples of 2^-54 E and the sines of 2^-55, E the power of two above the
# row's peak, and a sum is kept to 2^-52 E: with every rounding at its most 5 units of 2^-53 E for four terms,
# and as independent errors a sixth of 2.5 sqrt(H) units for H terms; the result's own rounding comes to that
@pytest.mark.parametrize("m,n", [(8, 12), (60, 8), (64, 36), (72, 8), (1000, 8), (1024, 8), (1080, 8), (2048, 8),
                                 (2160, 8)])
def test_transform_against_extended_precision(m, n):
    rng = np.random.default_rng(m)
    x = np.concatenate([_rows(k, n // 4, m, rng) for k in KINDS])
    g = _sim(m, n)
    y = g.pressure_transform(x)
    g.close()
    pick = np.arange(n) if m < 500 else np.arange(0, n, 2)   # the extended-precision sums are slow
    exact = x[pick].astype(LD) @ _sines(m)
    E = 2.0 ** np.ceil(np.log2(np.abs(x[pick]).max(axis=1)))[:, None]
    assert (np.abs((y[pick] - exact).astype(np.float64))
            <= 2.0 ** -53 * (np.abs(exact) + 2.5 * np.sqrt(m / 2) * E).astype(np.float64)).all()


@pytest.mark.parametrize("m", [800, 1200])
def test_error_is_no_larger_than_the_fp64_product(m):
    """The product in FP64, each output one chain of multiply-adds over the samples in order."""
    n = 16
    rng = np.random.default_rng(m)
    x = np.concatenate([_rows(k, n // 4, m, rng) for k in KINDS])
    g = _sim(m, n)
    y = g.pressure_transform(x)
    g.close()
    S = _sines(m)
    exact = x.astype(LD) @ S
    W = S.astype(np.float64).astype(LD)
    p = np.zeros((n, m))
    for j in range(m):
        p = (p + x[:, j:j + 1].astype(LD) * W[j]).astype(np.float64)
    for i, kind in enumerate(KINDS):
        r = slice(i * n // 4, (i + 1) * n // 4)
        here, fp64 = (float(np.linalg.norm((a[r] - exact[r]).astype(np.float64))) for a in (y, p))
        assert here <= fp64, kind


# half lines of one and of three chunks
@pytest.mark.parametrize("m", [64, 2160])
def test_transform_exponents(m):
    """A power of two factors out exactly, zeros stay zeros, results past the range become infinite or
    subnormal; a row with a sample that is not finite is NaN and no other row is."""
    n = 8
    x = np.random.default_rng(7).standard_normal((n, m))
    g = _sim(m, n)
    y = g.pressure_transform(x)
    for k in (-900, -300, 300, 900):
        assert np.array_equal(g.pressure_transform(x * 2.0 ** k), y * 2.0 ** k)
    mixed = 2.0 ** np.array([-900, 900, 0, -300, 300, 0, 1, -1])[:, None]
    assert np.array_equal(g.pressure_transform(x * mixed), y * mixed)
    assert not g.pressure_transform(np.zeros_like(x)).any()
    small = g.pressure_transform(x * 2.0 ** -1060)   # m samples rounded to 2^-1074, and the result
    assert np.isfinite(small).all() and np.abs(small - y * 2.0 ** -1060).max() <= (m + 1) * 5e-324
    assert np.isinf(g.pressure_transform(np.full_like(x, 1e308))).any()
    for bad in (np.nan, np.inf):
        z = x.copy()
        z[3, 7] = bad
        w = g.pressure_transform(z)
        assert np.isnan(w[3]).all()
        assert np.array_equal(np.delete(w, 3, 0), np.delete(y, 3, 0))
    g.close()


def test_timing_of_the_transform_that_runs():
    g = _sim(128, 64)
    assert g.time_pass(6, 3) > 0.0
    with pytest.raises(G.IbError, match="ARG"):
        g.time_pass(7, 3)
    g.close()
