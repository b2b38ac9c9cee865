"""Steepest descent with the stopping test on the device: iterations enqueued
past the stopping one change nothing, whatever its place among those enqueued
together."""
import ctypes
import time

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


MESH = (512, 512, 4)


def _tilted():
    """A film magnetised uniformly away from its easy axis: the torque falls from
    the first iterations on."""
    cfg = random_config(21, *MESH, "", terms=("exch", "anis", "demag"), spatial=False, holes=False)
    cfg.update(Ms=np.full(cfg["Ms"].size, 5e5), axis=(0, 0, 1), m=np.tile([0.4, 0.1, 0.9], cfg["Ms"].size))
    cfg["m"] /= np.linalg.norm(cfg["m"][:3])
    return cfg


def _timed(max_steps, stop, reps):
    """(iterations, max dm/dt, shortest time) of a descent on fresh handles."""
    cfg = _tilted()
    best = 1e9
    for _ in range(reps):
        g = GpuSim(cfg)
        g.field()
        g.h.call("mm_synchronize")
        n, mx = ctypes.c_int64(), ctypes.c_double()
        t = time.perf_counter()
        g.h.call("mm_relax", 0, max_steps, stop, ctypes.byref(n), ctypes.byref(mx))
        best = min(best, time.perf_counter() - t)
        g.h.close()
    return n.value, mx.value, best


def test_converged_descent_costs_one_iteration():
    """A descent whose first iteration meets the criterion runs that one only
    (512 x 512 x 4 FP64: 0.34 ms, and the call's allocations)."""
    _timed(1, 0.0, 1)
    n, _, stop = _timed(60, 1e12, 6)
    assert n == 1
    assert stop <= 1.5 * _timed(1, 0.0, 6)[2]


def test_iterations_past_the_stop_do_no_work():
    """512 x 512 x 4 FP64: the field kernel and the direct z transform are 0.13 of
    an iteration's 0.33 ms; the launches of one that returns at once take 0.02."""
    g = GpuSim(_tilted())
    n, mx, curve = ctypes.c_int64(), ctypes.c_double(), []
    for _ in range(140):  # the descent goes on from call to call
        g.h.call("mm_relax", 0, 1, 0.0, ctypes.byref(n), ctypes.byref(mx))
        curve.append(mx.value)
    # iterations 6 to 13, 14 to 21, ... are enqueued together: a stop early in one
    n = next(k for k in range(6, 140) if (k - 6) % 8 < 4 and curve[k - 1] < min(curve[:k - 1]))
    stop = curve[n - 1] * (1 + 1e-9)
    got, _, stopped = _timed(200, stop, 6)
    assert got == n
    assert stopped - _timed(n, 0.0, 6)[2] <= 0.06e-3 * (7 - (n - 6) % 8) + 0.05e-3
