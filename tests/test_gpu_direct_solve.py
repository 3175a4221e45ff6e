"""The stationary bodies' direct solve (products with the inverse Cholesky factor) against the oracle's
factorisation, over numbers of unknowns about the kernels' strides (a warp, four warps, a CTA's rows)."""
import pytest

from helpers import SMALL, pair, rel
from ib_parallel_gb300 import geometry as GEO

pytestmark = pytest.mark.gpu


# points at least one grid spacing apart: condition below 1e5, so a step agrees to 1e-10 (round-off
# 1e-16 times the condition, with a factor 10 left)
@pytest.mark.parametrize("m,npts", [(64, 2), (64, 15), (64, 16), (64, 17), (128, 33), (128, 64), (128, 65), (128, 98)])
def test_direct_solve_sizes(m, npts):
    kw = dict(SMALL, m=m, n=m // 2, num_stat=True)
    o, g = pair(kw, [GEO.cylinder(npts, diameter=2.0, xc=1.0)])
    for _ in range(2):
        o.advance()
        g.advance()
    assert rel(g.get_vector("f"), o.f) < 1e-10
    assert rel(g.get_field("omega", 0), o.omega[0]) < 1e-10
    g.close()
