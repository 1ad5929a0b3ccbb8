"""Storage order for numberings that do and do not run through space."""
import numpy as np
import pytest

from tests._support import gpu_domain, oracle_domain, rel_l2, rows
from weldform_gb300 import PRECISION_FP64, PRECISION_MIXED, configs

pytestmark = pytest.mark.gpu


def _renumbered(d, run, **kw):
    """The upset cylinder with its lattice numbered in runs of `run` particles
    taken in random order (0: as generated)."""
    add = d.AddCylinderLength

    def wrapped(*a):
        add(*a)
        if run:
            x = d.get_array("x")
            c = np.arange(len(x)) // run
            p = np.random.default_rng(5).permutation(c.max() + 1)
            d.set_array("x", x[np.argsort(p[c], kind="stable")])

    d.AddCylinderLength = wrapped
    return configs.cylinder_upsetting(d, R=0.006, L=0.012, dx=0.0005, jitter_amp=0.0, **kw)


@pytest.mark.parametrize("run,cells", [(0, 0), (32, 0), (16, 0), (4, 1), (2, 1), (1, 1)])
def test_the_rule_follows_the_numbering(run, cells):
    d = gpu_domain()
    c = _renumbered(d, run)
    d.prepare(c.dt)
    assert d.geti("cell_order") == cells
    d.close()


def _upset(x):
    return x * [1.0, 1.01, 0.96]


def _crushed(x):
    """Bricks of more particles than the shared-memory sort takes."""
    return x * [40.0, 1.0, 0.5]


@pytest.mark.parametrize("move", [_upset, _crushed])
@pytest.mark.parametrize("run", [1, 4])
def test_rows_in_cell_order_match_the_oracle(run, move):
    got = []
    for d in (gpu_domain(), oracle_domain()):
        c = _renumbered(d, run)
        d.prepare(c.dt)
        d.set_array("x", move(d.get_array("x")))
        d.neighbour_search()
        got.append(rows(*d.neighbours()))
        d.close()
    assert got[0] == got[1]


@pytest.mark.parametrize("precision,tol", [(PRECISION_FP64, 1e-9), (PRECISION_MIXED, 1e-4)])
def test_a_yielding_run_of_shuffled_particles_follows_the_oracle(precision, tol):
    """Rebuilds and filters in cell order; the forms' stated accuracies."""
    out = []
    for d in (gpu_domain(), oracle_domain()):
        if not out:
            d.set("precision", precision)
        c = _renumbered(d, 1, v_top=-20.0)
        d.prepare(c.dt)
        d.step(25)
        out.append({f: d.get_array(f) for f in ("x", "Sigma", "pl_strain")})
        assert d.geti("nb_searches") > 2
        d.close()
    assert out[1]["pl_strain"].max() > 0
    for f in out[0]:
        assert rel_l2(out[0][f], out[1][f]) <= tol, f
