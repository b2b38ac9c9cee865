"""The demag passes on compile-time line lengths: fields at the edges of their
ranges (smallest lines, odd cell counts, the largest two- and three-stage
lengths, columns that pass the product through shared memory, tiles that
straddle planes) against the CPU oracle; the run-time-length passes on meshes
that take the compile-time ones by default; and steepest descents, whose FP64
films keep the run-time arithmetic."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

from helpers import GpuSim, build_oracle, random_config, rel_maxnorm

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PATHS = [ROOT, os.path.join(ROOT, "micromagnetic.jl_b200"), os.path.dirname(os.path.abspath(__file__))]


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


# x: 8 .. 1301, y: 8 .. 4000 (film columns of 16 .. 8000; the FP64 form's of
# more than 2000 cells take the global-memory stages), z: 2 .. 128 cells; z = 16
# and 2 .. 5 go on to the register and the direct z convolution
MESHES = [(8, 1030, 1, ""), (1031, 8, 1, ""), (257, 33, 1, "x"), (9, 2048, 1, ""), (1301, 13, 1, ""), (150, 151, 1, ""),
          (97, 89, 6, ""), (33, 17, 72, "z"), (21, 10, 128, ""), (8, 700, 7, "y"), (129, 65, 2, ""), (300, 8, 10, ""), (8, 1600, 1, ""), (9, 1700, 1, "x"), (8, 1900, 1, ""),
          (8, 2000, 1, ""), (9, 2100, 1, ""), (8, 2560, 1, ""), (9, 3001, 1, "y"), (8, 4000, 1, ""), (40, 21, 16, ""),
          (50, 37, 5, "")]


@pytest.mark.parametrize("mesh", MESHES)
def test_fields_against_oracle(mesh):
    cfg = random_config(77 + mesh[0], *mesh, terms=("exch", "demag"))
    o, _ = build_oracle(cfg)
    ref = o.effective_field()
    assert rel_maxnorm(GpuSim(cfg, form=0).field(), ref) <= 1e-12
    assert rel_maxnorm(GpuSim(cfg, form=1).field(), ref) <= 1e-5


def _child(code, env):
    r = subprocess.run([sys.executable, "-c", "import sys; sys.path[:0] = %r\n" % (PATHS,) + code],
                       env=dict(os.environ, **env), capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout + r.stderr


RUNTIME = """
import numpy as np
from helpers import GpuSim, random_config
out = {}
for i, mesh in enumerate(%r):
    cfg = random_config(60 + i, *mesh, terms=("exch", "demag"), spatial=False)
    for form in (0, 1):
        g = GpuSim(cfg, form=form)
        out["h%%d_%%d" %% (i, form)] = g.field()
        g.rk4(2e-14, 2)
        out["m%%d_%%d" %% (i, form)] = g.m()
np.savez(%r, **out)
"""
# film columns within the tile budget, filling one block (FP64 1200, FP32 2600
# points) and in global-memory stages (FP64 2600); leftover columns of a
# power-of-two z convolution; other z lengths; wide and narrow row tiles; the
# register z convolutions on column-major spectra (FP64: lines past the last ky,
# every block full)
RUNTIME_MESHES = [(100, 82, 1), (40, 600, 1), (24, 1300, 1), (64, 10, 16), (97, 89, 6), (33, 17, 72), (130, 300, 3),
                  (64, 500, 16), (32, 1024, 16), (40, 900, 16)]


def test_run_time_passes_against_oracle(tmp_path):
    """MMCUDA_RFFT=0: the passes that film descents, the persistent step and meshes
    without a compile-time length run, on meshes that exercise their routes."""
    path = str(tmp_path / "runtime.npz")
    _child(RUNTIME % (RUNTIME_MESHES, path), {"MMCUDA_RFFT": "0"})
    got = np.load(path)
    for i, mesh in enumerate(RUNTIME_MESHES):
        o, _ = build_oracle(random_config(60 + i, *mesh, terms=("exch", "demag"), spatial=False))
        ref = o.effective_field()
        o.rk4(2e-14, 2)
        for form, tol_h, tol_m in ((0, 1e-12, 1e-11), (1, 1e-5, 1e-5)):
            assert rel_maxnorm(got[f"h{i}_{form}"], ref) <= tol_h, (mesh, form)
            assert rel_maxnorm(got[f"m{i}_{form}"], o.get_m()) <= tol_m, (mesh, form)


# FP64 films whose padded lengths agree with the run-time passes' and whose do
# not (a second plan), and a box, on the compile-time passes
@pytest.mark.parametrize("mesh", [(128, 80, 1), (101, 97, 1), (30, 18, 17)])
def test_descent_against_oracle(mesh):
    """Three and six iterations from a random state.  The Barzilai-Borwein quotients
    amplify rounding (by 1e8 in six iterations of the second film), so the
    bound is the oracle's own: a change of the exchange constant by 1e-14 moves its
    state by d, and the fields compared are good to 1e-12."""
    cfg = random_config(8 + mesh[0], *mesh, terms=("exch", "anis", "demag"), spatial=False)
    for steps in (3, 6):
        ref = []
        for eps in (0.0, 1e-14):
            o, _ = build_oracle(dict(cfg, A=cfg["A"] * (1 + eps)))
            o.relax("SD", steps, 0.0)
            ref.append(o.get_m())
        g = GpuSim(cfg)
        n, mx = ctypes.c_int64(), ctypes.c_double()
        g.h.call("mm_relax", 0, steps, 0.0, ctypes.byref(n), ctypes.byref(mx))
        assert n.value == steps
        assert rel_maxnorm(g.m(), ref[0]) <= 100 * rel_maxnorm(ref[1], ref[0]) + 1e-12


DESCENT = """
import ctypes
import numpy as np
from helpers import GpuSim, random_config
cfg = random_config(5, 101, 97, 1, terms=("exch", "anis", "demag"))
g = GpuSim(cfg, form=0)
n, mx = ctypes.c_int64(), ctypes.c_double()
g.h.call("mm_relax", 0, 40, 0.0, ctypes.byref(n), ctypes.byref(mx))
np.save(%r, g.m())
"""


def test_descent_keeps_the_run_time_arithmetic(tmp_path):
    """An FP64 film's descent gives the same bits with the compile-time passes
    on and off (its step lengths amplify rounding)."""
    out = []
    for flag in ("1", "0"):
        path = str(tmp_path / f"m{flag}.npy")
        _child(DESCENT % path, {"MMCUDA_RFFT": flag})
        out.append(np.load(path))
    np.testing.assert_array_equal(out[0], out[1])
