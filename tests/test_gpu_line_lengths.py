"""The demag passes on compile-time line lengths: fields at the edges of their
ranges (smallest lines, odd cell counts, the largest two- and three-stage
lengths, tiles that straddle planes) against the CPU oracle, and the
steepest descent of an FP64 film whose padded lengths differ from the
run-time passes'."""
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


# x: 8 .. 1301, y: 8 .. 2048 (film columns of 16 .. 4096), z: 6 .. 128 cells
MESHES = [(8, 1030, 1, ""), (1031, 8, 1, ""), (257, 33, 1, "x"), (9, 2048, 1, ""), (1301, 13, 1, ""), (150, 151, 1, ""),
          (97, 89, 6, ""), (33, 17, 72, "z"), (21, 10, 128, ""), (8, 700, 7, "y"), (129, 65, 2, ""), (300, 8, 10, "")]


@pytest.mark.parametrize("mesh", MESHES)
def test_fields_against_oracle(mesh):
    cfg = random_config(77 + mesh[0], *mesh, terms=("exch", "demag"))
    o, _ = build_oracle(cfg)
    ref = o.effective_field()
    assert rel_maxnorm(GpuSim(cfg, form=0).field(), ref) <= 1e-12
    assert rel_maxnorm(GpuSim(cfg, form=1).field(), ref) <= 1e-5


CHILD = """
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
        r = subprocess.run([sys.executable, "-c", "import sys; sys.path[:0] = %r\n" % (PATHS,) + CHILD % path],
                           env=dict(os.environ, MMCUDA_RFFT=flag), capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stdout + r.stderr
        out.append(np.load(path))
    np.testing.assert_array_equal(out[0], out[1])
