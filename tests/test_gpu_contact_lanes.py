"""One rigid plane's contact pass (several lanes per particle) against the oracle."""
import numpy as np
import pytest

from tests._support import gpu_domain, oracle_domain, rel_l2
from weldform_gb300 import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stiffness,friction,slide", [("wang", 0.0, 0.0), ("wang", 0.6, 0.0), ("area", 0.2, 5.0),
                                                      ("penalty", 0.2, 5.0)])
@pytest.mark.parametrize("R,L,dx", [(0.002, 0.003, 0.0005), (0.006, 0.004, 0.0004), (0.012, 0.002, 0.0002)],
                         ids=["wide_groups", "middle", "four_lanes"])
def test_plane_contact_matches_the_oracle(stiffness, friction, slide, R, L, dx):
    """1 and 12 steps from engaged contact in the plain form: contact rows equal, and
    state, contact forces, sums and the count of dynamic-friction evaluations
    as the oracle's serial walk gives them (1e-9, the plain form's bar).  The
    lattice is not jittered, so projections fall on edges shared by triangles."""
    def state(d):
        return dict(off=d.contact_pairs()[0], idx=d.contact_pairs()[1], v=d.get_array("v"), a=d.get_array("a"),
                    cf=d.get_array("contforce"), F=d.contact_force(0),
                    sums=np.array([d.get("contact_force_sum"), d.get("ext_forces_work")]),
                    dyn=d.geti("dynamic_friction_count"))

    out = []
    for d in (gpu_domain(), oracle_domain()):
        case = configs.contact_upsetting(d, R=R, L=L, dx=dx, v_punch=-10.0, friction=friction, stiffness=stiffness,
                                         v_slide=slide, thermal=False, jitter_amp=0.0, gap=-0.3 * dx)
        d.prepare(case.dt)
        d.step(1)
        first = state(d)
        d.step(11)
        out.append((first, state(d)))
        d.close()
    assert np.abs(out[1][0]["cf"]).max() > 0 and out[1][0]["off"][-1] > 0
    for g, o in zip(*out):
        assert np.array_equal(g["off"], o["off"]) and np.array_equal(g["idx"], o["idx"])
        assert g["dyn"] == o["dyn"]
        for k in ("v", "a", "cf", "F", "sums"):
            assert rel_l2(g[k], o[k]) <= 1e-9, k
