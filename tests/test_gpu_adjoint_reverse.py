"""The reverse step's kernels where their sizes can go wrong: one level (no ring passed on) to four,
vertex counts that are no multiple of a CTA's share, more bodies than one (the force coefficients'
layout), a first step alone (its right-hand sides merge); against the oracle's adjoint.  And the
checkpoint and tape arrays, which a context keeps for its next forward of a like size."""
import numpy as np
import pytest

import ib_adjoint as A
import ib_oracle as O
from ib_parallel_gb300 import ibgpu as G

pytestmark = pytest.mark.gpu


def _sims(m, n, levels, bodies=1):
    kw = dict(m=m, n=n, mgridlev=levels, dt=0.01, Re=100.0, len=4.0, offsetx=1.0, offsety=2.0 * n / m, num_stat=True,
              motion=(-1.0, 0.0, 0.0, 0.3, 0.0), autotune=False)
    cyl = [O.cylinder(npts=12, diameter=0.5, xc=0.3 + 0.9 * b, yc=0.0) for b in range(bodies)]
    p = O.Params(**{k: v for k, v in kw.items() if k in O.Params.__dataclass_fields__})
    return G.Simulation(G.Params(**kw), [G.Body(x=b.x.copy(), y=b.y.copy(), fam=1) for b in cyl]), O.IBOracle(p, cyl)


def _coefs(N, seed=0):
    t = np.arange(N, dtype=np.float64) + seed
    return np.stack([-1.0 + 0.1 * np.sin(t), 0.2 * np.cos(t), 0.3 * np.sin(0.5 * t)], 1)


# forces and gradient within the bounds the gradient test of the 64 x 32 cylinder holds (1e-10, 1e-9)
@pytest.mark.parametrize("m,n,levels,bodies,N", [(64, 32, 1, 1, 3), (60, 36, 2, 2, 4), (72, 40, 4, 1, 3), (80, 48, 2, 1, 1)])
def test_gradient_matches_the_oracle_adjoint(m, n, levels, bodies, N):
    g, o = _sims(m, n, levels, bodies)
    W = np.random.default_rng(m).standard_normal((N, bodies, 2))
    ad = A.Adjoint(o)
    Fo = ad.forward(_coefs(N))
    go = ad.backward(W)
    Fg = g.adjoint_forward(_coefs(N), K=2)
    gg = g.adjoint_backward(W)
    assert np.abs(Fg - Fo).max() < 1e-10 * np.abs(Fo).max()
    assert np.abs(gg - go).max() < 1e-9 * np.abs(go).max()


def test_kept_checkpoints_do_not_change_a_later_pass():
    passes = [(6, 2), (5, 2), (6, 3), (1, 1), (9, 4)]   # shorter, other segments, far smaller, larger
    g, _ = _sims(64, 32, 3)
    ref, _ = _sims(64, 32, 3)
    for i, (N, K) in enumerate(passes):
        W = np.random.default_rng(i).standard_normal((N, 1, 2))
        F = g.adjoint_forward(_coefs(N, i), K=K)
        grad = g.adjoint_backward(W)
        assert np.array_equal(F, ref.adjoint_forward(_coefs(N, i), K=N))
        assert np.array_equal(grad, ref.adjoint_backward(W)), i
