"""Checkpoints copied in one launch and reads through kept staging."""
import numpy as np
import pytest

from tests._support import gpu_domain
from weldform_gb300 import PRECISION_FP64, PRECISION_MIXED, configs

pytestmark = pytest.mark.gpu

FIELDS = ("x", "v", "a", "Sigma", "Strain_pl", "Density", "pl_strain", "T", "TIR", "Displacement")


def _state(d):
    out = {f: d.get_array(f) for f in FIELDS}
    out["Nb"] = d.get_array("Nb")
    out["off"], out["idx"] = d.neighbours()
    return out


@pytest.mark.parametrize("precision", [PRECISION_FP64, PRECISION_MIXED])
@pytest.mark.parametrize("case", ["yielding", "contact", "tensile_odd"])
def test_rewound_runs_repeat_bit_for_bit(precision, case):
    """Odd particle counts (columns off the 16-byte grid), row lengths from
    surface to interior, contact rows and the tensile columns."""
    d = gpu_domain()
    d.set("precision", precision)
    if case == "contact":
        c = configs.contact_upsetting(d, R=0.003, L=0.006, dx=0.0005, v_punch=-20.0, gap=-0.0001)
    else:
        c = configs.cylinder_upsetting(d, R=0.003, L=0.0056 if case == "tensile_odd" else 0.006, dx=0.0005, v_top=-20.0)
    if case == "tensile_odd":
        d.set_particles("TI", 0.3)
        d.set_particles("TIInitDist", c.dx)
    d.prepare(c.dt)
    d.step(8)
    start = _state(d)
    d.checkpoint_save(3)
    d.step(13)
    once = _state(d)
    for _ in range(2):
        d.checkpoint_restore(3)
        back = _state(d)
        for k in start:
            assert np.array_equal(start[k], back[k], equal_nan=True), k
        d.step(13)
        again = _state(d)
        for k in once:
            assert np.array_equal(once[k], again[k], equal_nan=True), k
    d.close()


def test_slot_saved_in_one_form_and_continued_in_the_other():
    """A slot saved by the plain form holds no mixed records: the mixed form
    continued from it builds them, as it does when it starts from that state."""
    runs = []
    for rewind in (False, True):
        d = gpu_domain()
        c = configs.cylinder_upsetting(d, R=0.003, L=0.006, dx=0.0005, v_top=-20.0)
        d.prepare(c.dt)
        d.step(6)
        d.checkpoint_save(0)
        d.set("precision", PRECISION_MIXED)
        if rewind:
            d.step(4)
            d.checkpoint_restore(0)
        d.step(5)
        runs.append(_state(d))
        d.close()
    for k in runs[0]:
        assert np.array_equal(runs[0][k], runs[1][k], equal_nan=True), k


def test_reads_and_writes_of_growing_and_shrinking_fields():
    d = gpu_domain()
    c = configs.cylinder_upsetting(d, R=0.002, L=0.004, dx=0.0005)
    d.prepare(c.dt)
    d.step(3)
    first = {f: d.get_array(f) for f in ("Density", "x", "Sigma", "Nb", "RotationRate", "pl_strain")}
    for f in reversed(list(first)):
        assert np.array_equal(first[f], d.get_array(f))
    d.set_array("T", np.arange(c.n, dtype=float))
    assert np.array_equal(d.get_array("T"), np.arange(c.n, dtype=float))
    assert np.array_equal(first["Sigma"], d.get_array("Sigma"))
    d.close()
