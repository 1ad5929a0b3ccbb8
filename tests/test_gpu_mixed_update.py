"""The mixed form's per-particle update: integer-pipe conversions, shared block
sums and the fused rate-stress kernel with the thermal solver."""
import numpy as np
import pytest

from tests._support import gpu_domain, oracle_domain, rel_l2
from weldform_gb300 import JOHNSON_COOK, PRECISION_MIXED, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("contact", [False, True])
def test_fused_rate_stress_with_the_thermal_solver_is_bit_identical(contact):
    """The same sums, update and block partials as k_rate_mx and k_stress_mx."""
    fields = ("x", "v", "Sigma", "pl_strain", "T", "dTdt", "Density", "StrainRate", "dint_energy_dt", "q_plheat")
    res = []
    for fuse in (0, 1):
        d = gpu_domain()
        d.set("precision", PRECISION_MIXED)
        if contact:
            case = configs.contact_upsetting(d, R=0.003, L=0.006, dx=0.0003, v_punch=-10.0, stiffness="area")
        else:
            case = configs.cylinder_upsetting(d, R=0.003, L=0.006, dx=0.0003, v_top=-20.0, model=JOHNSON_COOK,
                                              thermal=True)
        d.prepare(case.dt)
        d.set("gather_lanes", 1)
        d.set("fuse_rate_stress", fuse)
        d.step(40)
        assert ("k_rate_stress_mx" in d.profile_steps(1)) == bool(fuse)
        out = {f: d.get_array(f) for f in fields}
        for k in ("int_energy_sum", "kin_energy_sum", "plastic_work", "max_pl_strain", "m_maxT", "m_minT"):
            out[k] = d.get(k)
        res.append(out)
        d.close()
    assert res[0]["pl_strain"].max() > 0
    for k in res[0]:
        assert np.array_equal(res[0][k], res[1][k]), k


@pytest.mark.parametrize("block", [64, 128, 256])
@pytest.mark.parametrize("thermal", [False, True])
def test_block_sums_and_extremes(block, thermal):
    """Energy sums and the plastic-strain and temperature extremes over a last
    block that is nearly empty, against the oracle: the sums add FP32 pair
    sums' values (1e-5), the extremes are single particles' values (1e-5)."""
    out = []
    for d in (gpu_domain(), oracle_domain()):
        if not out:
            d.set("precision", PRECISION_MIXED)
            d.set("particle_block", block)
        case = configs.cylinder_upsetting(d, R=0.003, L=0.0061, dx=0.0005, v_top=-20.0, model=JOHNSON_COOK,
                                          thermal=thermal)
        T = np.full(case.n, 300.0)
        T[7], T[case.n - 1] = 290.0, 333.0  # the extremes sit in the first and in the last block
        d.set_array("T", T)
        d.prepare(case.dt)
        d.step(20)
        keys = ("int_energy_sum", "max_pl_strain") + (("plastic_work", "m_maxT", "m_minT") if thermal else ())
        out.append({k: d.get(k) for k in keys})
        d.close()
    assert out[1]["max_pl_strain"] > 0
    for k in out[1]:
        assert abs(out[0][k] - out[1][k]) <= 1e-5 * max(abs(out[1][k]), 1e-300), (k, out)


@pytest.mark.parametrize("scale", [0.0, 1e-45, 1e-39, 1e-30, 1e-12, 1.0, 1e3])
def test_velocity_scales_through_the_conversions(scale):
    """Zero, denormal and ordinary velocities through the float-float split and
    the widened rates: the mixed form follows the oracle at every scale that
    FP32 holds (1e-5: a few FP32 roundings of terms that cancel tenfold), and
    a body at rest stays exactly at rest."""
    out = []
    for d in (gpu_domain(), oracle_domain()):
        if not out:
            d.set("precision", PRECISION_MIXED)
        case = configs.cylinder_upsetting(d, R=0.003, L=0.006, dx=0.0005, v_top=0.0, jitter_amp=1e-3)
        rng = np.random.default_rng(3)
        v = rng.uniform(-1.0, 1.0, (case.n, 3)) * scale
        v[::3] = 0.0
        v[1::7] *= -1e-4
        d.set_array("v", v)
        d.prepare(case.dt)
        d.step(2)
        out.append((d.get_array("Displacement"), d.get_array("Sigma"), d.get_array("v")))
        d.close()
    for a, b in zip(*out):
        assert np.isfinite(a).all()
        if scale == 0.0:
            assert not a.any() and not b.any()
        elif scale >= 1e-12:
            assert rel_l2(a, b) <= 1e-5
