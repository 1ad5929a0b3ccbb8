"""The adjoint kernels with one, two and four lanes per particle give one gradient."""
import numpy as np
import pytest

from tests._support import gpu_domain
from weldform_gb300 import adjoint

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dx,thermal,slide", [(0.0012, True, 5.0), (0.0008, True, 0.0), (0.0008, False, 5.0),
                                              (0.0007, True, 0.0)], ids=["four", "two", "two_no_heat", "one"])
def test_gradient_against_central_differences(dx, thermal, slide):
    """dL/dPFAC and dL/dA by the adjoint against central differences of the loss
    at relative step 1e-5 over 12 steps (1e-3: the bar of the larger cases;
    the differences' own rounding is 1e-16 / 1e-5 of the loss, far below)."""
    case = adjoint.ContactCase(R=0.010, L=0.030, dx=dx, thermal=thermal, v_slide=slide, v_punch=-20.0)
    steps, every = 12, 4
    th = case.nominal()

    def domain(theta):
        d = gpu_domain()
        mesh = adjoint.build(d, case, theta)
        d.prepare(case.dt)
        return d, mesh

    d, mesh = domain(th)
    target = 0.9 * adjoint.reaction_curve(d, steps, every, mesh)
    d.close()
    d, mesh = domain(th)
    g = d.adjoint_reaction_loss(steps, every, target, mesh=mesh, checkpoint_every=5)
    d.close()
    for p in (9,) if not thermal else (9, 3):  # PFAC; A acts once particles yield
        loss = []
        for s in (1.0, -1.0):
            t = th.copy()
            t[p] *= 1.0 + s * 1e-5
            e, m = domain(t)
            loss.append(np.mean((adjoint.reaction_curve(e, steps, every, m) - target) ** 2))
            e.close()
        fd = (loss[0] - loss[1]) / (2e-5 * th[p])
        scale = max(abs(fd), 1e-6 * g["loss"] / th[p])
        assert abs(g["grad"][p] - fd) <= 1e-3 * scale, (p, g["grad"][p], fd)


@pytest.mark.parametrize("dx", [0.0012, 0.0008, 0.0007], ids=["four", "two", "one"])
def test_gradient_with_unequal_lengths_and_conductivities(dx):
    """Pairs whose smoothing lengths and conductivities differ, within warps whose
    other pairs agree: dL/dPFAC against central differences, the bar as above."""
    case = adjoint.ContactCase(R=0.010, L=0.030, dx=dx, thermal=True, v_punch=-20.0)
    steps, every = 12, 4
    th = case.nominal()

    def domain(theta):
        d = gpu_domain()
        mesh = adjoint.build(d, case, theta)
        few = np.random.default_rng(2).random(d.particle_count) < 0.02
        for f, s in (("h", 1.03), ("k_T", 1.5)):
            v = d.get_array(f)
            d.set_array(f, np.where(few, s * v, v))
        d.prepare(case.dt)
        return d, mesh

    d, mesh = domain(th)
    target = 0.9 * adjoint.reaction_curve(d, steps, every, mesh)
    d.close()
    d, mesh = domain(th)
    g = d.adjoint_reaction_loss(steps, every, target, mesh=mesh, checkpoint_every=5)
    d.close()
    loss = []
    for s in (1.0, -1.0):
        t = th.copy()
        t[9] *= 1.0 + s * 1e-5
        e, m = domain(t)
        loss.append(np.mean((adjoint.reaction_curve(e, steps, every, m) - target) ** 2))
        e.close()
    fd = (loss[0] - loss[1]) / (2e-5 * th[9])
    assert abs(g["grad"][9] - fd) <= 1e-3 * max(abs(fd), 1e-6 * g["loss"] / th[9])
