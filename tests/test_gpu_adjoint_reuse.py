"""Gradients of one handle called again and again: repeated backward calls
(segments replayed as graphs from the second one on), changed parameters,
checkpoint spacings and step counts, and segments without kept stage values,
against a handle that records once."""
import os
import subprocess
import sys

import numpy as np
import pytest

from helpers import GpuSim

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PATHS = [ROOT, os.path.join(ROOT, "micromagnetic.jl_b200"), os.path.dirname(os.path.abspath(__file__))]
DT = 5e-14


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _cfg(mesh=(24, 20, 2), seed=104):
    rng = np.random.default_rng(seed)
    n = mesh[0] * mesh[1] * mesh[2]
    m = rng.normal(size=(n, 3))
    m /= np.linalg.norm(m, axis=1, keepdims=True)
    return dict(nx=mesh[0], ny=mesh[1], nz=mesh[2], dx=2e-9, dy=2e-9, dz=2e-9, pbc="", Ms=rng.uniform(6e5, 9e5, n),
                m=m.reshape(-1), terms=["exch", "dmi_int", "anis", "demag"], A=1.3e-11,
                Dint=rng.uniform(1e-3, 4e-3, n), Ku=rng.uniform(2e5, 5e5, n), axis=(0, 0, 1), alpha=0.1, gamma=2.211e5)


def _backward(g, cfg, nsteps, ckpt):
    g.h.set_m(cfg["m"])
    g.h.call("mm_adjoint_record", DT, nsteps, ckpt)
    out = [np.zeros(3 * g.n)] + [np.zeros(g.n) for _ in range(3)]
    dp = g.lib.dptr
    w = np.random.default_rng(9).normal(size=3 * g.n)
    g.h.call("mm_adjoint_backward", dp(w), *(dp(o) for o in out))
    return out + [g.m()]


def _set_Ms(g, Ms):
    g.h.call("mm_set_Ms", g.lib.dptr(np.ascontiguousarray(Ms)), 0.0)


# (scale of Ms, steps, checkpoint spacing): the same call three times, other last
# segments with the same full ones, one segment a record, a segment longer than
# the replayed ones
CALLS = [(1.0, 24, 10), (1.0, 24, 10), (1.0, 24, 10), (1.0, 26, 10), (1.0, 26, 10), (1.0, 24, 10), (1.01, 24, 10),
         (1.01, 24, 10), (1.01, 20, 10), (1.01, 20, 10), (1.01, 7, 10), (1.01, 7, 10), (1.0, 70, 70), (1.0, 70, 70),
         (1.0, 24, 10), (1.0, 24, 10)]


@pytest.mark.parametrize("form", [0, 1])
def test_repeated_calls_equal_a_fresh_handle(form):
    cfg = _cfg()
    g = GpuSim(cfg, form=form)
    fresh, scale = {}, 1.0
    for call in CALLS:
        if call not in fresh:
            f = GpuSim(dict(cfg, Ms=cfg["Ms"] * call[0]), form=form)
            fresh[call] = _backward(f, cfg, *call[1:])
            f.h.close()
        if call[0] != scale:
            scale = call[0]
            _set_Ms(g, cfg["Ms"] * scale)
        for a, b in zip(_backward(g, cfg, *call[1:]), fresh[call]):
            np.testing.assert_array_equal(a, b)


def _instantiations(fn):
    """cudaGraphInstantiate calls made by fn."""
    from torch.profiler import ProfilerActivity, profile

    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
        fn()
    names = [e.name for e in prof.events()]
    if not any(n.startswith("cudaGraphLaunch") for n in names):  # a record's steps are graph launches
        pytest.skip("the profiler records no runtime calls here")
    return sum(n.startswith("cudaGraphInstantiate") for n in names)


def test_graphs_are_captured_for_reuse_only():
    """A loop that changes a parameter, the step count or the spacing before each
    record captures no segment (only the RK4 step after a changed parameter);
    a repeated record captures its two segment lengths once."""
    cfg = _cfg()
    g = GpuSim(cfg)
    for n in (23, 24):
        _backward(g, cfg, n, 10)

    def change(i):
        _set_Ms(g, cfg["Ms"] * (1 + 1e-3 * i))
        _backward(g, cfg, 24, 10)

    assert _instantiations(lambda: [change(i) for i in range(4)]) == 4
    assert _instantiations(lambda: [_backward(g, cfg, 23 + i % 3, 10) for i in range(6)]) == 0
    assert _instantiations(lambda: [_backward(g, cfg, 25, 10) for _ in range(6)]) == 2
