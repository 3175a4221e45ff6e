"""A step whose FSI iteration ends without a number reports IB_ERR_NONFINITE, whichever body the residual
without a number belongs to, with the iterations on the device and on the host."""
from dataclasses import replace

import numpy as np
import pytest

from helpers import PLATE, small_plate
from ib_parallel_gb300 import geometry as GEO
from ib_parallel_gb300 import ibgpu as G

pytestmark = pytest.mark.gpu

KW = dict(PLATE, n=64, offsetx=1.5, offsety=2.0, gmres_max_it=2000)


def _at(body, y):
    return replace(body, y=np.asarray(body.y) + y)


BODIES = {
    "plate": [small_plate()],
    "plates": [_at(small_plate(), -0.4), _at(small_plate(), 0.4)],
    "beam": [GEO.beam_plate(9, 1.0, 10.0, 0.5, 1e-2)],
    "beam and plate": [_at(GEO.beam_plate(9, 1.0, 10.0, 0.5, 1e-2), -0.4), _at(small_plate(), 0.4)],
    "rigid and beam": [GEO.cylinder(6, diameter=0.3, xc=1.0, yc=0.5),
                       _at(GEO.beam_plate(9, 1.0, 10.0, 0.5, 1e-2), -0.4)],
}


@pytest.mark.parametrize("bodies", list(BODIES))
@pytest.mark.parametrize("loop", ["device", "host"])
@pytest.mark.parametrize("where", ["omega", "f"])
def test_residual_without_a_number_is_reported(bodies, loop, where):
    g = G.Simulation(G.Params(**KW), BODIES[bodies])
    if loop == "host":
        g.step_profile(1)   # times the phases: the host runs the iterations
    for _ in range(3):
        g.advance()
    assert (g.step_graph_stats()["graph"] > 0) == (loop == "device")
    if where == "omega":
        g.set_field("omega", 0, np.full_like(g.get_field("omega", 0), np.nan))
    else:
        g.set_vector("f", np.full(g.nf, np.nan))   # the solve's initial guess
    with pytest.raises(G.IbError, match="NONFINITE"):
        g.advance()
    g.close()
