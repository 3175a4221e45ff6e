"""The cluster GMRES where its layout changes with the number of unknowns: slices without rows, a row
segment a lane in registers, rows in shared memory, more than eight blocks a slice, rows left in global
memory; against the graph solver, whose sums run one thread each in the same order, and the assembled
matrix."""
import numpy as np
import pytest

from ib_parallel_gb300 import ibgpu as G

pytestmark = pytest.mark.gpu

RTOL = 1e-6


def _sim(npts, plates, mode):
    d = 0.0625
    p = G.Params(m=256, n=128, mgridlev=2, dt=0.004, Re=100.0, len=16.0, offsetx=2.0, offsety=4.0, rtol=RTOL, atol=0.0,
                 fsi_tol=1e-9, autotune=False, schur_mode=mode)
    x = 2.0 * d * np.arange(npts) + 0.3 * d   # two spacings apart, off the grid lines
    bodies = [G.Body(x=x.copy(), y=np.full(npts, (i - 0.5 * (plates - 1)) * 16.0 * d + 0.2 * d), fam=1)
              for i in range(plates)]
    return G.Simulation(p, bodies)


@pytest.mark.parametrize("npts,plates", [(2, 1), (9, 1), (33, 1), (40, 2), (40, 4), (40, 6)])
def test_cluster_solver_matches_the_graph_solver(npts, plates):
    nf = 2 * npts * plates
    rng = np.random.default_rng(nf)
    b, x0 = rng.standard_normal(nf), 0.1 * rng.standard_normal(nf)
    out = []
    for mode in (0, 2):
        g = _sim(npts, plates, mode)
        S = g.schur_matrix()
        assert S is not None
        x, its = g.schur_solve(b, x0)
        assert its > 0
        # the residual estimate the solver stops at is the true residual's to one per cent
        assert np.linalg.norm(b - S @ x) <= 1.01 * RTOL * np.linalg.norm(b)
        out.append((x, its))
        g.close()
    assert out[0][1] == out[1][1]
    assert np.array_equal(out[0][0], out[1][0])
