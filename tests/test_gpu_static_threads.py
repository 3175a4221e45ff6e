"""ib_ctci_static set up for one grid after another on one thread, while others create contexts and step them:
its set-up ends no graph capture of theirs, and every result is the one of a thread alone."""
import threading

import numpy as np
import pytest

from helpers import PLATE, small_plate
from ib_parallel_gb300 import ibgpu as G

pytestmark = pytest.mark.gpu

GRIDS = [(64, 32), (120, 36), (96, 48), (200, 100)]


def _step():
    g = G.Simulation(G.Params(**dict(PLATE, autotune=False)), [small_plate()])
    for _ in range(4):
        g.advance()
    out = [g.get_field("omega", 0), g.get_vector("f")]
    g.close()
    return out


def test_static_setup_beside_stepping_threads():
    import torch

    rng = np.random.default_rng(5)
    stream = torch.cuda.Stream()
    data = [torch.from_numpy(rng.standard_normal((n - 1, m - 1))).cuda() for m, n in GRIDS]
    outs = [torch.zeros_like(d) for d in data]
    torch.cuda.synchronize()

    def solves():   # each call after the first on its grid is preceded by another grid's: all set up anew
        got = []
        for (m, n), d, s in zip(GRIDS, data, outs):
            G.ctci_static(m, n, d.data_ptr(), s.data_ptr(), stream.cuda_stream)
            with torch.cuda.stream(stream):
                got.append(s.cpu().numpy().copy())
        return got

    want, want_step = solves(), _step()
    failed, stop = [], threading.Event()

    def stepping():
        try:
            for _ in range(6):
                if not all(np.array_equal(a, b) for a, b in zip(_step(), want_step)):
                    failed.append("a step differs")
        except Exception as e:
            failed.append(repr(e))

    def solving():
        try:
            while not stop.is_set():
                if not all(np.array_equal(a, b) for a, b in zip(solves(), want)):
                    failed.append("a solve differs")
        except Exception as e:
            failed.append(repr(e))

    steppers = [threading.Thread(target=stepping) for _ in range(3)]
    solver = threading.Thread(target=solving)
    for t in steppers + [solver]:
        t.start()
    for t in steppers:
        t.join()
    stop.set()
    solver.join()
    assert not failed
