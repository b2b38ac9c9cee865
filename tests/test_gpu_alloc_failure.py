"""Device allocations that fail: a gradient, a descent and a demag plan go on
with what the handle can hold.  A preloaded stand-in of cudaMalloc returns
cudaErrorMemoryAllocation for requests above a limit that the child process
sets; no memory is exhausted."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PATHS = [ROOT, os.path.join(ROOT, "micromagnetic.jl_b200"), os.path.dirname(os.path.abspath(__file__))]

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
static size_t limit = (size_t)-1;
static long failed;
void fake_limit(size_t n) { limit = n; }
long fake_failed(void) { return failed; }
int cudaMalloc(void** p, size_t n) {
  static int (*real)(void**, size_t);
  if (!real) real = (int (*)(void**, size_t))dlsym(dlopen("libcudart.so.12", RTLD_NOLOAD | RTLD_LAZY), "cudaMalloc");
  if (n > limit) {
    ++failed;
    return 2;
  }
  return real(p, n);
}
"""

HEAD = """
import ctypes, sys
sys.path[:0] = %r
import numpy as np
from helpers import GpuSim, random_config
fake = ctypes.CDLL(None)
fake.fake_limit.argtypes = [ctypes.c_size_t]
fake.fake_failed.restype = ctypes.c_long
""" % (PATHS,)


@pytest.fixture(scope="module")
def child(tmp_path_factory):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    d = tmp_path_factory.mktemp("fake_alloc")
    (d / "shim.c").write_text(SHIM)
    so = str(d / "shim.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", so, str(d / "shim.c"), "-ldl"], check=True)

    def run(code, **env):
        """Runs code with the fake in place; it leaves its results in the dict `out`."""
        path = str(d / "out.npz")
        r = subprocess.run([sys.executable, "-c", HEAD + code + f"\nnp.savez({path!r}, **out)\n"],
                           env=dict(os.environ, LD_PRELOAD=so, **env), capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stdout + r.stderr
        return dict(np.load(path))

    return run


def close(a, b, tol):
    assert np.max(np.abs(a - b)) <= tol * np.max(np.abs(b))


GRAD = """
cfg = random_config(3, 24, 20, 2, terms=("exch", "dmi_int", "anis", "demag"), holes=False)
out = {}
for limit in (2**62, 1 << 20):  # the segment's stage values take 2.5 MB
    g = GpuSim(cfg, form=0)
    g.h.call("mm_adjoint_record", 5e-14, 20, 10)
    for call in range(3):
        fake.fake_limit(limit)
        o = [np.zeros(3 * g.n)] + [np.zeros(g.n) for _ in range(3)]
        g.h.call("mm_adjoint_backward", g.lib.dptr(np.ones(3 * g.n)), *(g.lib.dptr(x) for x in o))
        fake.fake_limit(2**62)
        for k, x in enumerate(o):
            out["%d_%d_%d" % (limit > 1 << 20, call, k)] = x
    out["failed%d" % (limit > 1 << 20)] = np.array(fake.fake_failed())
"""


def test_gradient_without_room_for_stage_values(child):
    """Both ways evaluate the same stages, the slopes by two kernels whose
    roundings differ: 20 steps of FP64 agree to 1e-11."""
    r = child(GRAD)
    assert r["failed1"] == 0 and r["failed0"] == 3  # asked for again by every call
    for call in range(3):
        for k in range(4):
            np.testing.assert_array_equal(r[f"0_{call}_{k}"], r[f"0_0_{k}"])
            close(r[f"0_{call}_{k}"], r[f"1_{call}_{k}"], 1e-11)


@pytest.mark.parametrize("env", [{"MMCUDA_ADJ_STORE": "0"}, {"MMCUDA_ADJ_KEEP_MB": "0"}])
def test_gradient_keeps_no_stage_values(child, env):
    """Switched off, and given back after every call."""
    a, b = child(GRAD, **env), child(GRAD)
    for call in range(3):
        for k in range(4):
            close(a[f"1_{call}_{k}"], b[f"1_{call}_{k}"], 1e-11)


BYTES = """
cfg = random_config(3, 24, 20, 2, terms=("exch", "dmi_int", "anis", "demag"), holes=False)
g = GpuSim(cfg, form=0)
out = {"b": []}
for call in range(4):
    g.h.call("mm_adjoint_record", 5e-14, 20, 10)
    o = [np.zeros(3 * g.n)] + [np.zeros(g.n) for _ in range(3)]
    g.h.call("mm_adjoint_backward", g.lib.dptr(np.ones(3 * g.n)), *(g.lib.dptr(x) for x in o))
    out["b"].append(g.h.device_bytes())
"""


def test_large_stage_values_are_given_back(child):
    """Above the kept size a handle holds the values during the call only."""
    kept, given = child(BYTES)["b"], child(BYTES, MMCUDA_ADJ_KEEP_MB="0")["b"]
    assert len(set(kept)) == 1 and len(set(given)) == 1
    assert kept[0] - given[0] == 8 * 11 * 3 * 960 * 10


DESCENT = """
from oracle.oracle import demag_tensor
cfg = random_config(5, 101, 97, 1, terms=("exch", "anis", "demag"))
T = demag_tensor(101, 97, 1, cfg["dx"], cfg["dy"], cfg["dz"])
out = {}
for name, tensor in (("own", None), ("given", T)):
    for limit in (2**62, 300000):  # the second plan's spectra take 475 kB
        g = GpuSim(cfg, form=0, tensor=tensor)
        n, mx = ctypes.c_int64(), ctypes.c_double()
        for part in (2, 2):
            fake.fake_limit(limit)
            g.h.call("mm_relax", 0, part, 0.0, ctypes.byref(n), ctypes.byref(mx))
            fake.fake_limit(2**62)
        out["%s%d" % (name, limit < 2**62)] = g.m()
    out["failed_" + name] = np.array(fake.fake_failed())
"""


def test_descent_without_room_for_its_own_plan(child):
    """An FP64 film's descent takes the handle's own plan when its second one
    cannot be allocated.  The first steps: the step lengths have not yet
    amplified the rounding (1e-15) of the two transforms beyond 1e-11."""
    r = child(DESCENT)
    assert r["failed_own"] > 0 and r["failed_given"] > r["failed_own"]
    for name in ("own", "given"):
        close(r[name + "1"], r[name + "0"], 1e-11)


PLAN = """
cfg = random_config(4, 8, 13, 128, terms=("exch", "demag"))
out = {}
for form in (0, 1):
    w = 4 if form else 8
    GpuSim(cfg, form=form).h.close()  # the tile widths kept for this mesh are those of the other lengths
    fake.fake_limit(250000 * w)  # y spectrum: 1.20 MB (FP32) at the compile-time lengths, 0.69 at the others
    f = fake.fake_failed()
    g = GpuSim(cfg, form=form)
    fake.fake_limit(2**62)
    out["failed%d" % form] = np.array(fake.fake_failed() - f)
    out["field%d" % form] = g.field()
"""


def test_demag_without_room_for_the_longer_lines(child):
    """The compile-time lengths pad more; where their buffers do not fit, the
    plan takes the run-time lengths."""
    from helpers import build_oracle, random_config, rel_maxnorm

    r = child(PLAN)
    o, _ = build_oracle(random_config(4, 8, 13, 128, terms=("exch", "demag")))
    ref = o.effective_field()
    for form, tol in ((0, 1e-12), (1, 1e-5)):
        assert r[f"failed{form}"] > 0
        assert rel_maxnorm(r[f"field{form}"], ref) <= tol
