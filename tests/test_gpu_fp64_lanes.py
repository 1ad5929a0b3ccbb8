"""The plain form's gathers with one, two and four lanes per particle, in their
uniform-particle and general forms, against the oracle."""
import numpy as np
import pytest

from tests._support import gpu_domain, oracle_domain, rel_l2
from weldform_gb300 import JOHNSON_COOK, configs

pytestmark = pytest.mark.gpu

FIELDS = ("x", "v", "a", "Sigma", "Density", "pl_strain", "StrainRate", "RotationRate", "T")


def _run(d, feature, R, L, dx, steps):
    jc = feature in ("thermal", "conduction_pairs")
    case = configs.cylinder_upsetting(d, R=R, L=L, dx=dx, v_top=-20.0, thermal=jc,
                                      **({"model": JOHNSON_COOK} if jc else {}))
    rng = np.random.default_rng(11)
    d.set_array("v", rng.uniform(-1.0, 1.0, (case.n, 3)))
    if feature == "h_varies":
        d.set_array("h", case.h * rng.uniform(0.97, 1.0, case.n))
    elif feature == "alpha_varies":
        d.set_array("Alpha", rng.uniform(0.0, 1.0, case.n))
    elif feature == "beta":
        d.set_particles("Beta", 2.0)
    elif feature == "inviscid":
        d.set_particles("Alpha", 0.0)
    elif feature == "tensile":
        d.set_particles("TI", 0.3)
        d.set_particles("TIInitDist", dx)
    elif feature == "gradcorr":
        d.set("gradKernelCorr", 1)
    elif feature == "leapfrog":
        d.set("integrator", 1)
    elif feature == "conduction_pairs":
        d.set_array("k_T", rng.uniform(20.0, 60.0, case.n))
        d.set_array("T", rng.uniform(300.0, 400.0, case.n))
    d.prepare(case.dt)
    d.step(steps)
    out = {f: d.get_array(f) for f in FIELDS}
    out["sums"] = np.array([d.get(k) for k in ("int_energy_sum", "max_pl_strain")])
    d.close()
    return out


@pytest.mark.parametrize("feature", ["uniform", "h_varies", "alpha_varies", "beta", "inviscid", "tensile", "gradcorr",
                                     "leapfrog", "thermal", "conduction_pairs"])
@pytest.mark.parametrize("size", [(0.003, 0.0061, 0.0005, 64), (0.003, 0.0061, 0.0005, 256),
                                  (0.006, 0.0141, 0.00042, 64)], ids=["four_lanes", "one_lane", "two_lanes"])
def test_plain_form_lanes_match_the_oracle(feature, size):
    """6 yielding steps from random velocities: the plain form's bar, 1e-9."""
    R, L, dx, block = size
    g = gpu_domain()
    g.set("particle_block", block)
    res = [_run(d, feature, R, L, dx, 6) for d in (g, oracle_domain())]
    for f in res[1]:
        assert rel_l2(res[0][f], res[1][f]) <= 1e-9, f
