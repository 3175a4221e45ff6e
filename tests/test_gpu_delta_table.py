"""The delta function's polynomial table against the oracle's closed form, at points whose distances
to the grid lines run through the table's parts and onto their ends."""
import numpy as np
import pytest

from helpers import SMALL, pair, rel
from ib_parallel_gb300 import geometry as GEO

pytestmark = pytest.mark.gpu


# weights are products of two values within 1e-16 of the closed form's exact value over delta; the
# oracle's double evaluation of it cancels terms of order one to below that of the weights' (1e-15)
@pytest.mark.parametrize("shift", [0.0, 1.0 / 64.0, 0.3])
def test_weights_across_the_table(shift):
    o, g = pair(SMALL, [GEO.cylinder(33)])
    d = SMALL["len"] / SMALL["m"]
    x = d * (4.0 + (np.arange(33) + shift) / 32.0)      # every 1/32 of a cell, ends included
    y = d * (1.0 + (np.arange(33) * 7 % 33 + shift) / 33.0)
    xb, yb = np.r_[x, x], np.r_[y, y]
    o.xb, o.yb = xb.copy(), yb.copy()
    o.setup_reg()
    g.reg_prep(xb, yb)
    h = np.random.default_rng(3).standard_normal(66)
    for a, b in zip(g.reg(h), o.reg(h)):
        assert rel(a, b) < 2e-14
    g.close()
