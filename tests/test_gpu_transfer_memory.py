"""Reads and writes of particle arrays stage their data in memory that the
domain has from its prologue: the first of them allocates nothing."""
import numpy as np
import pytest

from tests._support import gpu_domain
from weldform_gb300 import configs

pytestmark = pytest.mark.gpu


def test_transfers_take_no_device_memory():
    torch = pytest.importorskip("torch")
    d = gpu_domain()
    c = configs.cylinder_upsetting(d, R=0.006, L=0.012, dx=0.00025)
    d.prepare(c.dt)
    d.step(1)
    free = torch.cuda.mem_get_info(0)[0]
    first = {}
    for f in ("Density", "v", "Sigma", "RotationRate", "Nb"):
        first[f] = d.get_array(f)
        assert torch.cuda.mem_get_info(0)[0] == free, f
    x = d.get_array("x")
    d.set_array("x", x)
    assert torch.cuda.mem_get_info(0)[0] == free
    d.neighbour_search()  # the staging is the search's scratch: neither disturbs the other
    for f in first:
        assert np.array_equal(first[f], d.get_array(f)), f
    assert np.array_equal(x, d.get_array("x"))
    d.close()
