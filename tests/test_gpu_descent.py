"""Steepest descent with the stopping test on the device: iterations enqueued
past the stopping one change nothing, whatever its place among those enqueued
together."""
import ctypes

import numpy as np
import pytest

from helpers import GpuSim, random_config

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _relax(cfg, form, max_steps, stop):
    g = GpuSim(cfg, form=form)
    n, mx = ctypes.c_int64(), ctypes.c_double()
    g.h.call("mm_relax", 0, max_steps, stop, ctypes.byref(n), ctypes.byref(mx))
    return n.value, mx.value, g.m()


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("mesh", [(96, 90, 1, ""), (12, 9, 4, "x")])
def test_stop_leaves_the_state_of_its_iteration(form, mesh):
    cfg = random_config(11, *mesh, terms=("exch", "anis", "demag"))
    curve = [_relax(cfg, form, k, 0.0) for k in range(14, 24)]  # every place in a group of eight
    assert [c[0] for c in curve] == list(range(14, 24))
    for n, mx, m in curve:
        got, mx2, m2 = _relax(cfg, form, 60, mx * (1 + 1e-9))
        # the first iteration below the threshold, at the latest this one
        assert got <= n and mx2 < mx * (1 + 1e-9)
        if got == n:
            assert mx2 == mx
            np.testing.assert_array_equal(m2, m)
        else:
            np.testing.assert_array_equal(m2, _relax(cfg, form, got, 0.0)[2])
    assert _relax(cfg, form, 0, 0.0)[0] == 0
