"""The compiled term sets of the stage kernels, and the two-cells-a-thread FP32
stage (2^18 cells and more, even nx; odd nx takes one cell a thread): FP32
against the FP64 form after two RK4 and two Heun steps, and all twelve sets
against the general kernel, the adaptive stages included.

Tolerance: a step rotates m by gamma |H| dt ~ 1e-2 with a field good to 1e-5
(the FP32 form's field tolerance), and the state carries a low part: 1e-6."""
import os
import subprocess
import sys

import numpy as np
import pytest

from helpers import GpuSim, random_config, rel_maxnorm

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


SETS = [("exch", "demag"), ("exch", "anis", "demag"), ("exch", "dmi_bulk", "anis", "demag"),
        ("exch", "dmi_int", "demag"), ("exch", "dmi_int", "anis", "demag")]
# pairs: 2^18 cells exactly, the last pair of a row alone in its block, one row
# a plane, periodic wraps; 513: odd nx
MESHES = [(512, 512, 1, ""), (258, 34, 30, "xyz"), (1026, 257, 1, "x"), (513, 512, 1, "y")]


@pytest.mark.parametrize("terms", SETS)
@pytest.mark.parametrize("mesh", MESHES)
def test_fp32_stage_against_fp64(mesh, terms):
    cfg = random_config(3 + mesh[0], *mesh, terms=terms, spatial=False)
    a, b = GpuSim(cfg, form=1), GpuSim(cfg, form=0)
    a.rk4(5e-14, 2)
    b.rk4(5e-14, 2)
    assert rel_maxnorm(a.m(), b.m()) <= 1e-6
    a.h.call("mm_heun_run", 1e-14, 2)
    b.h.call("mm_heun_run", 1e-14, 2)
    assert rel_maxnorm(a.m(), b.m()) <= 1e-6
    assert np.isfinite(a.m()).all()


ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PATHS = [ROOT, os.path.join(ROOT, "micromagnetic.jl_b200"), os.path.dirname(os.path.abspath(__file__))]
ALL_SETS = [("exch",) + dmi + anis + zee + ("demag",) for dmi in ((), ("dmi_bulk",), ("dmi_int",))
            for anis in ((), ("anis",)) for zee in ((), ("zeeman",))]
RUN = """
import sys
sys.path[:0] = %r
import numpy as np
from helpers import GpuSim, random_config
out = {}
for k, terms in enumerate(%r):
    for j, mesh in enumerate(((512, 512, 1, "x"), (21, 18, 23, "yz"))):  # two cells a thread in FP32; one
        for form in (0, 1):
            cfg = random_config(50 + k, *mesh, terms=[t for t in terms if t != "zeeman"], spatial=False)
            g = GpuSim(cfg, form=form)
            if "zeeman" in terms:
                g.h.call("mm_add_zeeman", None, 2e4, -1e4, 3e4)
            key = "%%d_%%d_%%d" %% (k, j, form)
            g.rk4(5e-14, 2)
            g.heun(1e-14, 2)
            out["fixed" + key] = g.m()
            rc, st = g.run_until(2e-13)
            out["steps" + key] = np.array([rc, st["nsteps"], st["attempts"]])
            out["adaptive" + key] = g.m()
            g.h.close()
np.savez(%r, **out)
"""


def test_compiled_sets_against_the_general_kernel(tmp_path):
    """MMCUDA_STAGE_FIX=0 evaluates the same sums in the general kernel; the
    compilers contract other multiply-adds: 1e-12 a field in FP64, 1e-6 in FP32
    (2e-13 s of an adaptive run: ten times that)."""
    out = []
    for flag in "10":
        path = str(tmp_path / f"fix{flag}.npz")
        r = subprocess.run([sys.executable, "-c", RUN % (PATHS, ALL_SETS, path)],
                           env=dict(os.environ, MMCUDA_STAGE_FIX=flag), capture_output=True, text=True, timeout=900)
        assert r.returncode == 0, r.stdout + r.stderr
        out.append(np.load(path))
    a, b = out
    assert len(ALL_SETS) == 12 and len(a.files) == 12 * 2 * 2 * 3
    for key in a.files:
        if key.startswith("steps"):
            assert a[key][0] == 0 and a[key][1] > 2
            np.testing.assert_array_equal(a[key], b[key], key)
            continue
        tol = (1e-12 if key.endswith("0") else 1e-6) * (10 if key.startswith("adaptive") else 1)
        assert rel_maxnorm(a[key], b[key]) <= tol, key
