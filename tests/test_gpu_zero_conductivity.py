"""Conduction between two particles of zero conductivity: the reference's
harmonic mean 4 k_i k_j / (k_i + k_j) is 0/0 there, and every form says so."""
import numpy as np
import pytest

from tests._support import gpu_domain, oracle_domain
from weldform_gb300 import JOHNSON_COOK, PRECISION_FP64, PRECISION_MIXED, configs

pytestmark = pytest.mark.gpu


def _dTdt(d, k_T, vary_h):
    c = configs.cylinder_upsetting(d, R=0.003, L=0.006, dx=0.0005, model=JOHNSON_COOK, thermal=True)
    k = np.full(c.n, 40.0)
    if k_T == "all_zero":
        k[:] = 0.0
    elif k_T == "half_zero":
        k[: c.n // 2] = 0.0
    elif k_T == "one_zero":
        k[c.n // 2] = 0.0
    d.set_array("k_T", k)
    if vary_h:  # not uniform: the general gathers
        d.set_array("h", d.get_array("h") * np.linspace(0.99, 1.0, c.n))
    d.set_array("T", 300.0 + np.arange(c.n) % 7)
    d.prepare(c.dt)
    d.step(1)
    out = d.get_array("dTdt")
    d.close()
    return out


@pytest.mark.parametrize("vary_h", [False, True])
@pytest.mark.parametrize("k_T", ["all_zero", "half_zero", "one_zero", "none_zero"])
@pytest.mark.parametrize("precision", [PRECISION_FP64, PRECISION_MIXED])
def test_the_same_particles_are_without_a_rate(precision, k_T, vary_h):
    d = gpu_domain()
    d.set("precision", precision)
    got, want = _dTdt(d, k_T, vary_h), _dTdt(oracle_domain(), k_T, vary_h)
    assert np.isnan(want).any() == (k_T in ("all_zero", "half_zero"))
    assert np.array_equal(np.isnan(got), np.isnan(want))
    # FP64: a sum of ~60 terms that cancel to about their own size (1e-12);
    # mixed: FP32 pair terms (1e-4, the form's stated accuracy)
    f = np.isfinite(want)
    tol = 1e-12 if precision == PRECISION_FP64 else 1e-4
    if f.any():
        assert np.abs(got[f] - want[f]).max() <= tol * np.abs(want[f]).max()
