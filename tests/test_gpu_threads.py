"""Contexts created, stepped and closed by several host threads at once give the results they give one after
another: no thread's set-up ends a graph capture of another's."""
import threading

import numpy as np
import pytest

from ib_parallel_gb300 import geometry as GEO
from ib_parallel_gb300 import ibgpu as G

pytestmark = pytest.mark.gpu

KINDS = ["plate", "beam", "cylinder", "sub-domain", "adjoint"]


def _run(i):
    kind, m = KINDS[i % len(KINDS)], [96, 128, 160, 200][i % 4]
    kw = dict(m=m, n=m // 2, mgridlev=1 + i % 3, dt=0.4 / m, Re=100.0, len=8.0, offsetx=2.0, offsety=2.0, fsi_tol=1e-9,
              atol=1e-13, rtol=1e-11, autotune=False, num_stat=kind in ("cylinder", "adjoint"))
    npts = m // 16 + 1
    body = {"beam": GEO.beam_plate(npts, 1.0, 10.0, 0.5, 1e-2), "cylinder": GEO.cylinder(npts),
            "adjoint": GEO.cylinder(npts)}.get(kind, GEO.torsional_plate(npts, 1.0, -10.0, itheta=0.5 / 3.0, ktheta=1e-2))
    g = G.Simulation(G.Params(**kw), [body])
    out = []
    if kind == "sub-domain":
        g.subdomain_setup(-0.5, 1.5, -0.6, 0.6, 8.0 / m)
    if kind == "adjoint":
        out += [g.adjoint_forward(np.tile([-1.0, 0.1, 0.02], (4, 1)), 2), g.adjoint_backward(np.ones((4, 1, 2)))]
    else:
        for _ in range(4):
            g.advance()
    out += [g.get_field("omega", k) for k in range(kw["mgridlev"])] + [g.get_vector("f")] + g.pressure()
    g.close()
    return out


def test_threads_give_the_sequential_results():
    n = 2 * len(KINDS)
    want = [_run(i) for i in range(n)]
    for _ in range(3):
        got, failed = [None] * n, []

        def work(i):
            try:
                got[i] = _run(i)
            except Exception as e:   # reported below: an exception in a thread fails no test by itself
                failed.append((i, repr(e)))

        threads = [threading.Thread(target=work, args=(i,)) for i in range(n)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not failed
        for a, b in zip(got, want):
            assert all(np.array_equal(x, y) for x, y in zip(a, b))
