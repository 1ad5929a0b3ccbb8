"""Checkpoints taken right after the prologue, before any search has filled the
superset: what lies in the memory then is not read as row lengths."""
import numpy as np
import pytest

from tests._support import gpu_domain
from weldform_gb300 import PRECISION_FP64, PRECISION_MIXED, configs

pytestmark = pytest.mark.gpu

FIELDS = ("x", "v", "Sigma", "Density", "pl_strain")


def _state(d):
    out = {f: d.get_array(f) for f in FIELDS}
    out["off"], out["idx"] = d.neighbours()
    return out


def _same(a, b):
    for k in a:
        assert np.array_equal(a[k], b[k], equal_nan=True), k


def _leave_used_memory():
    """A domain whose supersets and rows are filled, closed again: the next
    domain's allocations may get its memory."""
    d = gpu_domain()
    c = configs.cylinder_upsetting(d, R=0.006, L=0.012, dx=0.0004, v_top=-20.0)
    d.prepare(c.dt)
    d.step(8)
    d.close()


def _prepared(precision):
    d = gpu_domain()
    d.set("precision", precision)
    c = configs.cylinder_upsetting(d, R=0.004, L=0.008, dx=0.0005, v_top=-20.0)
    d.prepare(c.dt)
    return d


@pytest.mark.parametrize("precision", [PRECISION_FP64, PRECISION_MIXED])
def test_a_checkpoint_before_the_first_step_rewinds_to_it(precision):
    d = _prepared(precision)
    assert d.geti("skin_reuse") == 1
    d.step(5)
    want = _state(d)
    d.close()
    _leave_used_memory()
    d = _prepared(precision)
    d.checkpoint_save(0)
    d.step(5)
    _same(want, _state(d))
    d.checkpoint_restore(0)
    d.step(5)
    _same(want, _state(d))
    d.close()


def test_autotuning_before_the_first_step_leaves_the_run_as_it_was():
    _leave_used_memory()
    d = _prepared(PRECISION_MIXED)
    d.autotune(2)
    block, lanes = d.geti("gather_block"), d.geti("gather_lanes")
    d.step(5)
    got = _state(d)
    d.close()
    d = _prepared(PRECISION_MIXED)
    d.set("gather_block", block)
    d.set("gather_lanes", lanes)
    d.step(5)
    _same(got, _state(d))
    d.close()
