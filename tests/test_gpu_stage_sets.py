"""The compiled term sets of the stage kernels, and the two-cells-a-thread FP32
stage (2^18 cells and more, even nx; odd nx takes one cell a thread): FP32
against the FP64 form after two RK4 and two Heun steps.

Tolerance: a step rotates m by gamma |H| dt ~ 1e-2 with a field good to 1e-5
(the FP32 form's field tolerance), and the state carries a low part: 1e-6."""
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
