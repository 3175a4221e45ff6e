"""The FSI iterations of beams on the device against the same iterations run from the host: the same
kernels' arithmetic, so the same steps bit for bit.  And the beam kernels where their row groups can go wrong: fewer DOFs than a group of lanes, more than a
pass of the CTA covers, elements longer than several points and shorter than one, two beams; the
structure operators against the oracle's dense formulation."""
import numpy as np
import pytest

from helpers import PLATE, pair, rel, small_plate
from ib_parallel_gb300 import geometry as GEO
from ib_parallel_gb300 import ibgpu as G
from dataclasses import replace

pytestmark = pytest.mark.gpu


def _beam(npts, nelem, y=0.0):
    b = GEO.beam_plate(npts, 1.0, 10.0, 0.5, 1e-2)
    return replace(b, nelem=nelem, y=np.asarray(b.y) + y)


# the forward error of a solve with K_eff (and the bounds of the beam operators' own test where larger)
@pytest.mark.parametrize("sizes", [[(3, 1)], [(9, 1)], [(9, 3)], [(9, 11)], [(33, 16)], [(79, 39)], [(7, 3), (12, 5)]])
def test_beam_operators(sizes):
    o, g = pair(PLATE, [_beam(npts, nelem, 0.4 * i) for i, (npts, nelem) in enumerate(sizes)])
    rng = np.random.default_rng(len(sizes) + sizes[0][0])
    tol = max([1e-12] + [b.ndof * 2.0**-52 * np.linalg.cond(b.Keff) for b in o.beams])
    for _ in range(2):
        f = 1e-2 * rng.standard_normal(o.nf)
        err_o = o.compute_dx(f)
        o.setup_reg()
        err_g = g.struct_dx(f)
        qo = np.concatenate([b.q for b in o.beams])
        qm = np.abs(qo).max()
        assert abs(err_g - err_o) <= tol * max(err_o, qm)
        assert rel(g.beam_state()[0], qo) < tol
        assert np.abs(g.get_vector("xb") - o.xb).max() < 1e-14 + tol * qm
        assert np.abs(g.get_vector("yb") - o.yb).max() < 1e-14 + tol * qm
        scale = o.delta * 2.0 / PLATE["dt"] * np.abs(qo).max()
        assert np.abs(g.struct_rhs() - o.compute_rhs()).max() < tol * scale
    g.close()


@pytest.mark.parametrize("beams,plate", [([(9, 0, 0.0)], False), ([(9, 3, -0.3), (7, 0, 0.3)], False), ([(9, 0, -0.3)], True)])
@pytest.mark.parametrize("subdomain", [False, True])
def test_device_iterations_match_the_host_loop(beams, plate, subdomain):
    bodies = [_beam(*b) for b in beams]
    if plate:   # a torsional body beside the beam: both errors join the loop's condition
        t = small_plate()
        bodies.append(replace(t, y=np.asarray(t.y) + 0.3))
    kw = dict(PLATE, n=64, offsetx=1.5, offsety=2.0)   # room for the sub-domain's cloud
    gd, gh = (G.Simulation(G.Params(**kw), bodies) for _ in range(2))
    if subdomain:
        for g in (gd, gh):
            g.subdomain_setup(-0.4, 1.4, -0.7, 0.6, PLATE["len"] / PLATE["m"])
    gh.step_profile(1)   # times the phases: the host runs the iterations
    for step in range(6):
        gd.advance()
        gh.advance()
        assert gd.counters() == gh.counters(), step
        for a, b in zip(gd.beam_state(), gh.beam_state()):
            assert np.array_equal(a, b), step
        assert np.array_equal(gd.get_vector("f"), gh.get_vector("f"))
        for k in range(PLATE["mgridlev"]):
            assert np.array_equal(gd.get_field("omega", k), gh.get_field("omega", k)), (step, k)
    assert gd.step_graph_stats()["graph"] >= 3 and gh.step_graph_stats()["graph"] == 0
    gd.close()
    gh.close()
