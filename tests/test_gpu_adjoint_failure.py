"""A forward of the adjoint whose later step fails: the coefficients of the steps before it are delivered, the
call reports the failure, and nothing is left to reverse."""
import numpy as np
import pytest

from helpers import SMALL, small_cylinder
from ib_parallel_gb300 import ibgpu as G

pytestmark = pytest.mark.gpu

IB_ERR_GMRES = 4


@pytest.mark.parametrize("K", [1, 2, 5])
def test_coefficients_before_a_failing_step(K):
    frames = np.tile([-1.0, 0.1, 0.02], (4, 1))
    kw = dict(SMALL, motion=(-1.0, 0.0, 0.0, 0.0, 0.0))
    g = G.Simulation(G.Params(**kw), [small_cylinder()])
    want = g.adjoint_forward(frames, K)
    g.close()
    frames[2] = np.nan   # no Krylov solve of this step converges
    g = G.Simulation(G.Params(**kw), [small_cylinder()])
    out = np.full((4, 1, 2), 7.0)
    rc = g.lib.ib_adjoint_forward(g.h, 4, K, G._ptr(frames), G._ptr(out))
    assert rc == IB_ERR_GMRES
    assert np.array_equal(out[:2], want[:2]) and (out[2:] == 7.0).all()
    with pytest.raises(G.IbError, match="STATE"):
        g.adjoint_backward(np.ones((4, 1, 2)))
    g.close()
