"""A restored checkpoint brings back the kernels and constants that its fields
select, whatever was written to h, Alpha, Beta, mass or Cs in between."""
import numpy as np
import pytest

from tests._support import gpu_domain
from weldform_gb300 import PRECISION_FP64, PRECISION_MIXED, configs

pytestmark = pytest.mark.gpu

FIELDS = ("x", "v", "Sigma", "Density", "pl_strain", "h", "Alpha", "Beta", "Mass", "Cs")


def _vary(a):
    return a * np.linspace(0.97, 1.0, len(a))


# what the saved state has, then what is written over it
BRANCHES = {
    "alpha_off": ({}, {"Alpha": lambda a: 0.0 * a}),
    "alpha_other": ({}, {"Alpha": lambda a: 0.25 * a}),
    "alpha_varying": ({}, {"Alpha": _vary}),
    "alpha_on": ({"Alpha": 0.0}, {"Alpha": lambda a: a + 1.0}),
    "beta_off": ({"Beta": 0.5}, {"Beta": lambda a: 0.0 * a}),
    "beta_on": ({}, {"Beta": lambda a: a + 0.5}),
    "h_other": ({}, {"h": lambda a: 0.95 * a}),
    "h_varying": ({}, {"h": _vary}),
    "h_uniform": ({"h": _vary}, {"h": lambda a: np.full_like(a, a.min())}),
    "mass_varying": ({}, {"Mass": _vary}),
    "cs_other": ({}, {"Cs": lambda a: 0.9 * a}),
    "cs_varying": ({}, {"Cs": _vary}),
}


def _domain(precision, first):
    d = gpu_domain()
    d.set("precision", precision)
    c = configs.cylinder_upsetting(d, R=0.003, L=0.006, dx=0.0005, v_top=-20.0)
    for f, v in first.items():
        if callable(v):
            d.set_array(f, v(d.get_array(f)))
        else:
            d.set_particles(f, v)
    d.prepare(c.dt)
    d.step(6)
    return d


def _after(d):
    d.step(6)
    out = {f: d.get_array(f) for f in FIELDS}
    out["uniform_layout"] = d.geti("uniform_layout")
    return out


@pytest.mark.parametrize("steps_between", [0, 3])
@pytest.mark.parametrize("branch", list(BRANCHES))
@pytest.mark.parametrize("precision", [PRECISION_FP64, PRECISION_MIXED])
def test_a_restored_state_steps_as_if_nothing_was_written(precision, branch, steps_between):
    first, write = BRANCHES[branch]
    d = _domain(precision, first)
    want = _after(d)
    d.close()
    d = _domain(precision, first)
    d.checkpoint_save(0)
    for f, change in write.items():
        d.set_array(f, change(d.get_array(f)))
    d.step(steps_between)
    d.checkpoint_restore(0)
    got = _after(d)
    d.close()
    for k in want:
        assert np.array_equal(want[k], got[k], equal_nan=True), k
