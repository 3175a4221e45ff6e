"""Body points far outside the sub-domain cloud, or not numbers: the interpolation takes the cloud's nearest
cell, whatever the distance, the call reports the domain, and the same context forms the same operator
afterwards."""
import numpy as np
import pytest

from helpers import PLATE, small_plate
from ib_parallel_gb300 import ibgpu as G

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def plate():
    g = G.Simulation(G.Params(**PLATE), [small_plate()])
    g.subdomain_setup(-0.25, 1.25, -0.25, 0.25, 0.0625)
    g.subdomain_precompute()
    yield g
    g.close()


@pytest.mark.parametrize("axis", ["x", "y"])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, 1e7, 1e9, 1e300, -1e300])
def test_points_out_of_the_clouds_reach(plate, bad, axis):
    g = plate
    xb, yb = g.get_vector("xb"), g.get_vector("yb")
    before = g.subdomain_operator()
    n = len(xb) // 2
    xs, ys = xb.copy(), yb.copy()
    v = ys if axis == "y" else xs
    v[n - 3:n] = v[2 * n - 3:] = bad   # the last three points
    with pytest.raises(G.IbError, match="DOMAIN"):
        g.reg_prep(xs, ys)
    with pytest.raises(G.IbError, match="DOMAIN"):
        g.subdomain_operator()
    g.reg_prep(xb, yb)
    assert np.array_equal(g.subdomain_operator(), before)
