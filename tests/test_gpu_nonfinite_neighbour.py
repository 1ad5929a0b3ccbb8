"""A pair at a non-finite distance has no kernel gradient (0, the branch that a
NaN takes in the reference's comparisons), in the uniform-particle gathers too."""
import numpy as np
import pytest

from tests._support import gpu_domain, oracle_domain

pytestmark = pytest.mark.gpu


def _strain_rate(d, side, vary_h):
    """One step in which one particle of a unit lattice drifts to infinity in x
    while its velocity, density and those of its neighbours stay finite."""
    r = 0.5
    d.AddBoxLength(0, (0.0, 0.0, 0.0), 6.0, 6.0, 6.0, r, 1e-8, 1.2, 1, 0, False, False)
    n = d.particle_count
    x = d.get_array("x")
    j = int(np.argmin(((x - x.mean(0)) ** 2).sum(1)))
    rng = np.random.default_rng(3)
    v = rng.uniform(-1e-12, 1e-12, (n, 3))
    v[j] = (side * 2e300, 0.0, 0.0)
    d.set_array("v", v)
    if vary_h:
        d.set_array("h", d.get_array("h") * np.linspace(0.999, 1.0, n))
    for f, val in (("G", 1.0), ("Cs", 1.0), ("Fail", 1), ("Sigmay", 1e300)):
        d.set_particles(f, val)
    d.prepare(1e8)
    d.step(1)
    out = d.get_array("StrainRate").reshape(n, 9)
    xn = d.get_array("x")
    d.close()
    assert not np.isfinite(xn[j, 0])
    return out


@pytest.mark.parametrize("vary_h", [False, True])
@pytest.mark.parametrize("side", [-1.0, 1.0])
def test_components_without_the_infinite_distance_stay_finite(side, vary_h):
    got, want = _strain_rate(gpu_domain(), side, vary_h), _strain_rate(oracle_domain(), side, vary_h)
    bad = np.isnan(want)
    yy = 4
    assert bad[:, 0].sum() > 20 and not bad[:, yy].all()
    assert (bad[:, 0] & ~bad[:, yy]).any()
    assert np.array_equal(bad, np.isnan(got))
