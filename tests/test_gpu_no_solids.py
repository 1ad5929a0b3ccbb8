"""A rigid plane without a solid particle: refused with the same words at the
prologue and at every step after it."""
import pytest

from tests._support import gpu_domain
from weldform_gb300 import PRECISION_FP64, PRECISION_MIXED, WFError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [PRECISION_FP64, PRECISION_MIXED])
def test_a_plane_alone_is_refused_alike_by_prologue_and_step(precision):
    d = gpu_domain()
    d.set("precision", precision)
    d.AddCylinderLength(0, (0.0, 0.0, 0.0), 0.0001, 0.004, 0.00025, 7850.0, 0.0006, False)  # thinner than a particle
    assert d.particle_count == 0
    d.set("contact", 1)
    for c in "xyz":
        d.set(f"DomMin.{c}", -0.01)
        d.set(f"DomMax.{c}", 0.01)
    d.add_rigid_plane(2, False, (-0.005, -0.005, 0.0), (0.005, 0.005, 0.0), 8, 10)
    assert d.particle_count > 0
    for call in (lambda: d.prepare(1e-8), lambda: d.step(1), lambda: d.step(1)):
        with pytest.raises(WFError, match="No external particles found"):
            call()
    d.close()
