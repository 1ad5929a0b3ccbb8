"""The storage order (bricks of cells, original order inside) leaves the rows as the oracle's."""
import numpy as np
import pytest

from tests._support import gpu_domain, oracle_domain, rel_l2, rows
from weldform_gb300 import PRECISION_MIXED, configs

pytestmark = pytest.mark.gpu


def _cylinder(d, move, dx=0.0005, R=0.006, L=0.012):
    """prepare() on the lattice, then positions moved by `move` and a full search."""
    case = configs.cylinder_upsetting(d, R=R, L=L, dx=dx)
    d.prepare(case.dt)
    x = d.get_array("x")
    d.set_array("x", move(x.copy()))
    d.neighbour_search()
    return d.neighbours()


def _out_of_grid(x):
    """Half of the body beyond the grid: it is binned into the clamped edge
    cells, whose bricks hold more particles than the shared-memory sort takes."""
    x[x[:, 2] > 0.006, 2] += 0.05
    return x


def _crushed(x):
    """Rows along x torn apart (most end up in the clamped edge cells) and the
    layers pushed together, ~45 neighbours in a particle's own y-z plane."""
    x[:, 0] *= 40.0
    x[:, 2] *= 0.5
    return x


@pytest.mark.parametrize("move", [lambda x: x, lambda x: x * [1.0, 1.01, 0.96], _out_of_grid, _crushed,
                                  lambda x: x[np.random.default_rng(5).permutation(len(x))]],
                         ids=["lattice", "upset", "out_of_grid", "crushed", "shuffled"])
def test_rows_after_moves_match_the_oracle(move):
    got = []
    for d in (gpu_domain(), oracle_domain()):
        got.append(rows(*_cylinder(d, move)))
        d.close()
    assert got[0] == got[1]


@pytest.mark.parametrize("box", [(0.004, 0.004, 0.004, 0), (0.02, 0.003, 0.003, 0), (0.003, 0.003, 0.02, 1)],
                         ids=["hcp", "hcp_long_x", "cubic_long_z"])
def test_box_rows_and_acceleration(box):
    """Other packings and aspect ratios: rows equal, and the mixed form's second
    acceleration within FP32 pair rounding of the oracle's (about 20 roundings
    of 6e-8 per pair term, and a sum that cancels to no less than a tenth of
    its terms' norm under random velocities and the stress they make: 1.2e-5)."""
    Lx, Ly, Lz, pack = box
    out = []
    for d in (gpu_domain(), oracle_domain()):
        d.set("precision", PRECISION_MIXED) if not out else None
        r = 0.00025
        d.AddBoxLength(0, (0.0, 0.0, 0.0), Lx, Ly, Lz, r, 7850.0, 1.2 * 2 * r, pack, 0, False, False)
        n = d.particle_count
        rng = np.random.default_rng(7)
        d.set_array("x", d.get_array("x") + rng.uniform(-1e-3, 1e-3, (n, 3)) * r)
        d.set_array("v", rng.uniform(-1.0, 1.0, (n, 3)))
        for f, v in (("G", 7.7e10), ("Cs", 4600.0), ("Alpha", 1.0), ("Beta", 0.5), ("Fail", 1), ("Sigmay", 3e8)):
            d.set_particles(f, v)
        d.prepare(2e-8)
        d.step(2)
        out.append((rows(*d.neighbours()), d.get_array("a")))
        d.close()
    assert out[0][0] == out[1][0]
    assert rel_l2(out[0][1], out[1][1]) <= 1.2e-5


@pytest.mark.parametrize("skin", [0, 1])
@pytest.mark.parametrize("hfac", [0.55, 0.7, 0.9, 1.2, 1.35])
def test_rows_over_cell_occupancies(hfac, skin):
    """From cells of one particle (more than 32 non-empty cells in a stencil,
    every candidate opening one) to cells of twenty (none opening in some
    rounds of 32), with and without the superset: rows equal to the oracle's."""
    out = []
    for d in (gpu_domain(), oracle_domain()):
        if not out:
            d.set_f64("nb_skin", 0.1 if skin else 0.0)
        r = 0.00025
        d.AddBoxLength(0, (0.0, 0.0, 0.0), 0.005, 0.004, 0.006, r, 7850.0, hfac * 2 * r, 1, 0, False, False)
        n = d.particle_count
        d.set_array("x", d.get_array("x") + np.random.default_rng(3).uniform(-0.1, 0.1, (n, 3)) * r)
        for f, v in (("G", 7.7e10), ("Cs", 4600.0), ("Fail", 1), ("Sigmay", 3e8)):
            d.set_particles(f, v)
        d.prepare(2e-8)
        d.set_array("x", d.get_array("x") * [1.0, 1.02, 0.97])
        d.neighbour_search()
        out.append(rows(*d.neighbours()))
        d.close()
    assert out[0] == out[1]
    assert sum(len(r) for r in out[0]) > 0
