"""The stationary bodies' direct solve against the substitutions with a Cholesky factor of the same matrix:
its residual and its error are no larger, at unknowns about the kernels' strides."""
import numpy as np
import pytest
import scipy.linalg as sla

from helpers import SMALL, small_plate
from ib_parallel_gb300 import geometry as GEO
from ib_parallel_gb300 import ibgpu as G

pytestmark = pytest.mark.gpu

LD = np.longdouble


@pytest.mark.parametrize("m,npts", [(64, 2), (64, 16), (128, 33), (128, 65), (128, 98), (256, 157)])
def test_residual_and_error_beside_substitution(m, npts):
    g = G.Simulation(G.Params(**dict(SMALL, m=m, n=m // 2, num_stat=True)), [GEO.cylinder(npts, diameter=2.0, xc=1.0)])
    nf = g.nf
    A = np.empty((nf, nf))
    for i in range(nf):
        A[:, i] = g.schur_apply(np.eye(nf)[i], with_b=False)
    A = np.triu(A) + np.triu(A, 1).T   # what is factored
    L = sla.cho_factor(A, lower=True)
    Al = A.astype(LD)
    rng = np.random.default_rng(npts)
    here, there = [], []
    for b in [A @ rng.standard_normal(nf) for _ in range(3)] + [rng.standard_normal(nf) for _ in range(3)]:
        exact = sla.cho_solve(L, b).astype(LD)
        for _ in range(4):
            exact = exact + sla.cho_solve(L, (b - Al @ exact).astype(np.float64))
        for out, x in ((here, g.direct_solve(b)), (there, sla.cho_solve(L, b))):
            out.append([np.linalg.norm((b - Al @ x).astype(np.float64)),
                        np.linalg.norm((x - exact).astype(np.float64))])
    g.close()
    here, there = np.array(here).sum(axis=0), np.array(there).sum(axis=0)
    assert here[0] <= there[0]   # the residual
    assert here[1] <= there[1]   # the error


def test_only_where_a_matrix_is_factored():
    g = G.Simulation(G.Params(**SMALL), [small_plate()])
    with pytest.raises(G.IbError, match="STATE"):
        g.direct_solve(np.zeros(g.nf))
    g.close()
