"""Searches of bodies that have left their grid: bricks taken in parts, and
cells of more particles than the shared-memory sort takes."""
import numpy as np
import pytest

from tests._support import gpu_domain, oracle_domain, rows
from weldform_gb300 import configs

pytestmark = pytest.mark.gpu

MOVES = {
    "x_out": lambda x: x + [0.05, 0.0, 0.0],
    "y_out": lambda x: x + [0.0, 0.05, 0.0],
    "z_out": lambda x: x + [0.0, 0.0, 0.05],      # every column of cells ends in its top cell
    "edge_out": lambda x: x + [0.0, 0.05, 0.05],  # cells of ~500 particles
    "corner_out": lambda x: x + 0.05,             # one cell holds them all
    "half_in_corner": lambda x: x + 0.05 * (np.arange(len(x))[:, None] % 2),
}


@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("move", list(MOVES))
def test_rows_of_bodies_out_of_the_grid_match_the_oracle(move, shuffled):
    got = []
    for d in (gpu_domain(), oracle_domain()):
        c = configs.cylinder_upsetting(d, R=0.006, L=0.012, dx=0.0005)
        if shuffled:
            x = d.get_array("x")
            d.set_array("x", x[np.random.default_rng(5).permutation(len(x))])
        d.prepare(c.dt)
        d.step(1)
        d.set_array("x", MOVES[move](d.get_array("x")))
        d.neighbour_search()
        got.append(rows(*d.neighbours()))
        d.set_array("x", d.get_array("x"))  # the counts are zero again for the search after it
        d.neighbour_search()
        got.append(rows(*d.neighbours()))
        d.close()
    assert got[0] == got[1] == got[2] == got[3]
    assert sum(len(r) for r in got[0]) > 0
