"""Restarted GMRES: several cycles of short restarts on both drivers, bit for bit and against the assembled
matrix, and the restarts of 33 to 60 vectors that the graph solver alone takes."""
import numpy as np
import pytest

from ib_parallel_gb300 import ibgpu as G

pytestmark = pytest.mark.gpu


def _solve(npts, spacing, restart, rtol, mode):
    d = 0.0625
    p = G.Params(m=256, n=128, mgridlev=2, dt=0.004, Re=100.0, len=16.0, offsetx=2.0, offsety=4.0, rtol=rtol, atol=0.0,
                 fsi_tol=1e-9, autotune=False, schur_mode=mode, gmres_restart=restart)
    x = spacing * d * np.arange(npts) + 0.3 * d   # off the grid lines
    g = G.Simulation(p, [G.Body(x=x, y=np.full(npts, 0.2 * d), fam=1)])
    rng = np.random.default_rng(restart)
    b, x0 = rng.standard_normal(g.nf), 0.1 * rng.standard_normal(g.nf)
    S = g.schur_matrix()
    f, its = g.schur_solve(b, x0)
    g.close()
    # the residual estimate the solver stops at is the true residual's to one per cent
    assert np.linalg.norm(b - S @ f) <= 1.01 * rtol * np.linalg.norm(b)
    return f, its


@pytest.mark.parametrize("restart", [1, 2, 5, 8])
@pytest.mark.parametrize("npts", [9, 33])
def test_short_restarts(restart, npts):
    (f0, n0), (f2, n2) = (_solve(npts, 2.0, restart, 1e-6, mode) for mode in (0, 2))
    assert n0 == n2 > restart
    assert np.array_equal(f0, f2)


# points five quarters of a spacing apart (condition 150): more vectors than any restart holds
@pytest.mark.parametrize("restart", [32, 33, 40, 60])
def test_long_restarts(restart):
    f, its = _solve(60, 1.25, restart, 1e-8, 0)
    assert its > restart
