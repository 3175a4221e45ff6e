"""The pressure's fixed-point x transform and the tridiagonal solve's chunkings at the sizes where they
can go wrong: half lines below, at and above a tile (32) and a summation chunk (512 terms), rows that
no equal chunking divides, and row counts past each chunk length."""
import numpy as np
import pytest

import ib_oracle as O
from helpers import SMALL, pair, rel
from ib_parallel_gb300 import ibgpu as G

pytestmark = pytest.mark.gpu


# tolerance: the level solves invert D D^T, whose lowest modes have condition (2 n_max / pi)^2, and
# ddti's transforms carry a few units of 1e-16 each
@pytest.mark.parametrize("m,n", [(8, 12), (20, 16), (60, 36), (64, 60), (72, 100), (128, 40), (1000, 16), (1200, 24)])
def test_pressure_sizes(m, n, tmp_path):
    kw = dict(SMALL, m=m, n=n, mgridlev=2)
    o, g = pair(kw, [])
    rng = np.random.default_rng(m + n)
    for k in range(2):
        g.set_field("omega", k, 0.1 * rng.standard_normal((n - 1, m - 1)))
        g.set_field("qx", k, rng.standard_normal((n, m + 1)))
        g.set_field("qy", k, rng.standard_normal((n + 1, m)))
    path = tmp_path / "data00.var"
    g.write_variables(path)
    O.restore(o, O.read_variables(path), itime=0)
    for a, b in zip(g.pressure(), o.calculate_pressure()):
        assert rel(a, b) < 1e-13 * max(10.0, (2 * max(m, n) / np.pi) ** 2 / 100.0)
    g.close()


# 539 rows: 14 chunks of 39, the last shorter; 1295: chunks of 63; 2159: the shared-memory kernel
@pytest.mark.parametrize("m,n", [(12, 540), (12, 1296), (8, 2160)])
def test_poisson_chunkings(m, n):
    o, g = pair(dict(SMALL, m=m, n=n, mgridlev=1), [])
    x = np.random.default_rng(n).standard_normal((n - 1, m - 1))
    assert rel(g.ctci(x), o.ctci(x)) < 1e-13 * (n / 100.0) ** 2
    g.close()
