"""Points that are not numbers or lie far outside the grid: their stencil origins stay near the grid, so that
the box of all stencils, which the contribution lists index, keeps a size that can be checked (unbounded, its
face count wrapped to a negative index beside a body inside).  The call reports the domain, and the same
context gives the same results afterwards."""
import numpy as np
import pytest

from helpers import PLATE, SMALL, rel, small_plate
from ib_parallel_gb300 import geometry as GEO
from ib_parallel_gb300 import ibgpu as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, 1e5, -1e5, 1e12, 1e300])
@pytest.mark.parametrize("axis", ["x", "y", "both"])
def test_points_out_of_reach_are_reported(bad, axis):
    bodies = [GEO.cylinder(8, diameter=0.5, xc=0.0), GEO.cylinder(7, diameter=0.5, xc=2.0)]
    g = G.Simulation(G.Params(**SMALL), bodies)
    xb, yb = g.get_vector("xb"), g.get_vector("yb")
    h = np.random.default_rng(3).standard_normal(len(xb))
    before = g.reg(h)
    xs, ys = xb.copy(), yb.copy()
    if axis != "y":
        xs[16:] = bad   # the second body's unknowns
    if axis != "x":
        ys[16:] = bad
    with pytest.raises(G.IbError, match="DOMAIN"):
        g.reg_prep(xs, ys)
    g.reg(h)
    g.redistribute(h)
    g.reg_prep(xb, yb)
    for a, b in zip(g.reg(h), before):
        assert np.array_equal(a, b)
    g.close()


def test_the_step_after_a_restore_is_not_blamed(tmp_path):
    """A step that ends without a number leaves its body nowhere; the restored context steps as before."""
    g = G.Simulation(G.Params(**PLATE), [small_plate()])
    for _ in range(3):
        g.advance()
    g.write_variables(tmp_path / "data00.var")
    g.advance()
    after = g.get_field("omega", 0)
    g.set_field("omega", 0, np.full_like(after, np.nan))
    with pytest.raises(G.IbError, match="NONFINITE"):
        g.advance()
    g.read_variables(tmp_path / "data00.var", 3)
    g.advance()
    assert rel(g.get_field("omega", 0), after) < 1e-8   # the restart test's bound
    g.close()
