"""E^T over boxes of every kind: one body's, whose faces nearly all have entries, two bodies near and a domain
apart, where a warp meets many empty faces; against the oracle."""
import numpy as np
import pytest

from helpers import SMALL, pair, rel
from ib_parallel_gb300 import geometry as GEO

pytestmark = pytest.mark.gpu


# tolerance: a face sums at most a few dozen products of weights that agree to 1e-14
@pytest.mark.parametrize("m,centres", [(64, [(1.0, 0.0)]), (64, [(0.0, 0.0), (4.0, 0.3)]), (320, [(1.0, 0.0)]),
                                       (320, [(-1.0, -1.0), (4.9, 1.1)]),
                                       (320, [(-1.0, 0.0), (0.0, 0.2), (4.9, -0.1)])])
def test_spread_over_boxes(m, centres):
    o, g = pair(dict(SMALL, m=m, n=m // 2), [GEO.cylinder(17, diameter=0.6, xc=x, yc=y) for x, y in centres])
    h = np.random.default_rng(m).standard_normal(g.nf)
    for a, b in zip(g.reg(h), o.reg(h)):
        assert rel(a, b) < 1e-13
    g.close()
