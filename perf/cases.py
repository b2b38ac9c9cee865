"""Performance cases of the finite-difference LLG path.

Each case is a simulation a user of the package runs: a mesh, a material, a
precision and an integrator, driven through the package's own API.  `listed()`
gives fixed cases from the smallest mesh to the largest, `draw()` further ones
of the same ranges; `prepare()` builds the simulation (terms, demag tensor,
initial state, pinned output buffers), `run()` is one pass of the user's loop
(some steps, then the magnetisation copied out), and `exact()` evaluates the
same pass in 64 bits with plain numpy / torch.

The initial states are smooth textures (a few long-wavelength modes) with a
small short-wavelength perturbation, the states such simulations start from
and pass through.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "micromagnetic.jl_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

MU0 = 4 * math.pi * 1e-7

# Material parameter sets: A (J/m), Ms (A/m), alpha, and the optional terms
# bulk DMI (J/m^2), interfacial DMI (J/m^2), uniaxial anisotropy along z
# (J/m^3), a uniform field (T), a spin-orbit torque (aj, bj, p); `disc` puts
# the magnet in an ellipse inscribed in the mesh (nonmagnetic corners) and
# `vary` draws Ms per cell.
MATERIALS = {
    "permalloy": dict(A=1.3e-11, Ms=8e5, alpha=0.02, B=(-0.0246, 0.0043, 0.0)),
    "block": dict(A=1.3e-11, Ms=8e5, alpha=0.1),
    "chiral": dict(A=1e-11, Ms=5.8e5, alpha=0.1, Dbulk=3e-3, Ku=5e5),
    "interface": dict(A=1.3e-11, Ms=7e5, alpha=0.1, Dint=3e-3, Ku=4e5, vary=True),
    "racetrack": dict(A=1.3e-11, Ms=8e5, alpha=0.1, Dint=2e-3, Ku=5e5, B=(0.0, 0.0, 0.02),
                      sot=(8e8, 2e8, (0.0, 1.0, 0.0))),
    "dot": dict(A=1.3e-11, Ms=8e5, alpha=0.05, disc=True, B=(0.01, 0.0, 0.0)),
}
GAMMA = 2.211e5


def listed():
    return [
        # the smallest everyday run: the standard-problem-4 film with the
        # default adaptive integrator, where launches and latency count
        dict(name="std4_dopri_f64", kind="dopri", form="f64", nx=200, ny=50, nz=1, dx=2.5, dy=2.5, dz=3.0,
             material="permalloy", span=4e-12),
        # an odd-sized track with interfacial DMI and a current: the torque terms
        dict(name="track_rk4_f32", kind="rk4", form="f32", nx=251, ny=93, nz=1, dx=2.0, dy=2.0, dz=1.0,
             material="racetrack", steps=100, dt=5e-14),
        # energy minimisation of an ultrathin chiral film (steepest descent)
        dict(name="film_relax_f64", kind="relax", form="f64", nx=320, ny=320, nz=1, dx=2.0, dy=2.0, dz=1.0,
             material="interface", steps=60),
        # the published film benchmark: Heun on 1000 x 1000
        dict(name="film1000_heun_f32", kind="heun", form="f32", nx=1000, ny=1000, nz=1, dx=4.0, dy=4.0, dz=4.0,
             material="permalloy", steps=40, dt=1e-14),
        # its large end: 16 million cells, the longest lines in common use
        dict(name="film4000_heun_f32", kind="heun", form="f32", nx=4000, ny=4000, nz=1, dx=4.0, dy=4.0, dz=4.0,
             material="permalloy", steps=6, dt=1e-14),
        # a thick elliptic element on an odd mesh, double precision
        dict(name="box_rk4_f64", kind="rk4", form="f64", nx=150, ny=126, nz=37, dx=3.0, dy=3.0, dz=3.0,
             material="dot", steps=10, dt=5e-14),
        # an ordinary multilayer-like mesh of no special size, single precision
        dict(name="box_rk4_f32", kind="rk4", form="f32", nx=300, ny=200, nz=20, dx=2.5, dy=2.5, dz=2.0,
             material="interface", steps=20, dt=5e-14),
        # a bulk chiral magnet with the default adaptive integrator
        dict(name="chiral_dopri_f32", kind="dopri", form="f32", nx=256, ny=256, nz=64, dx=2.0, dy=2.0, dz=2.0,
             material="chiral", span=2.5e-13),
        # the headline mesh in both precisions
        dict(name="block_rk4_f32", kind="rk4", form="f32", nx=1024, ny=1024, nz=16, dx=3.0, dy=3.0, dz=3.0,
             material="block", steps=10, dt=5e-14),
        dict(name="block_rk4_f64", kind="rk4", form="f64", nx=1024, ny=1024, nz=16, dx=3.0, dy=3.0, dz=3.0,
             material="block", steps=4, dt=5e-14),
        # an ensemble of uneven films stepped together
        dict(name="ensemble_rk4_f32", kind="batch", form="f32", count=24, lo=32, hi=256, zmax=4, shapes=103,
             material="interface", steps=40, dt=5e-14),
        # gradients of a loss on the final state with respect to the initial
        # state and the material parameters (forward and backward sweep)
        dict(name="grad_rk4_f64", kind="adjoint", form="f64", nx=128, ny=128, nz=4, dx=2.0, dy=2.0, dz=2.0,
             material="interface", steps=40, dt=5e-14, every=20),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: film, box, ensemble or gradient, sizes log-uniform."""
    kind = rng.choice(["film", "film", "film", "box", "box", "box", "batch", "adjoint"])
    form = rng.choice(["f32", "f32", "f64"])
    if kind == "batch":
        return dict(kind="batch", form=form, count=rng.randint(6, 24), lo=rng.randint(16, 48),
                    hi=rng.randint(96, 256), zmax=rng.randint(1, 4), shapes=rng.randint(1, 1 << 20),
                    material=rng.choice(["interface", "permalloy"]), steps=rng.randint(20, 40), dt=5e-14)
    if kind == "adjoint":
        return dict(kind="adjoint", form="f64", nx=_logint(rng, 24, 160), ny=_logint(rng, 24, 160),
                    nz=rng.randint(1, 6), dx=2.0, dy=2.0, dz=2.0, material="interface", steps=rng.randint(10, 30),
                    dt=5e-14, every=rng.choice([5, 10, 20]))
    if kind == "film":
        nx, ny, nz = _logint(rng, 32, 2200), _logint(rng, 32, 2200), 1
        integ = rng.choice(["rk4", "rk4", "heun", "dopri", "relax"])
        material = rng.choice(["permalloy", "interface", "racetrack", "dot"])
        dx, dz = rng.choice([2.0, 2.5, 4.0]), rng.choice([1.0, 2.0, 3.0])
    else:
        nz = _logint(rng, 2, 72)
        cap = 6e6 if form == "f64" else 1.2e7
        nx = _logint(rng, 24, 640)
        ny = min(_logint(rng, 24, 1024), max(24, int(cap / (nx * nz))))
        integ = rng.choice(["rk4", "rk4", "rk4", "heun", "dopri"])
        material = rng.choice(["block", "chiral", "interface", "dot"])
        dx, dz = rng.choice([2.0, 2.5, 3.0]), rng.choice([2.0, 3.0])
    if integ == "relax" and form == "f32":
        integ = "heun"  # descents are run in double precision
    n = nx * ny * nz
    case = dict(kind=integ, form=form, nx=nx, ny=ny, nz=nz, dx=dx, dy=dx, dz=dz, material=material)
    if integ == "dopri":
        case["span"] = 2e-12 if n < 2e5 else 2e-13
    elif integ == "relax":
        case["steps"] = rng.randint(20, 60)
    else:
        case.update(steps=max(4, min(80, int(6e7 / n))), dt=1e-14 if integ == "heun" else 5e-14)
    return case


# ------------------------------------------------------------------ inputs --
def _shapes(case):
    if case["kind"] != "batch":
        return [(case["nx"], case["ny"], case["nz"])]
    r = np.random.default_rng(case["shapes"])
    return [(int(r.integers(case["lo"], case["hi"] + 1)), int(r.integers(case["lo"], case["hi"] + 1)),
             int(r.integers(1, case["zmax"] + 1))) for _ in range(case["count"])]


def _texture(shape, seed):
    """Unit vectors (N, 3), cell index (k*ny + j)*nx + i: four long-wavelength
    modes per component plus 2 % of cell-scale noise."""
    nx, ny, nz = shape
    r = np.random.default_rng(seed)
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    f8 = dict(dtype=torch.float64, device="cuda")
    x = torch.arange(nx, **f8)[None, None, :] / max(nx, ny)
    y = torch.arange(ny, **f8)[None, :, None] / max(nx, ny)
    z = torch.arange(nz, **f8)[:, None, None] / max(nx, ny)
    out = torch.empty(nz, ny, nx, 3, **f8)
    for c in range(3):
        v = torch.full((1, 1, 1), float(r.normal()) * 0.5, **f8)
        for _ in range(4):
            kx, ky, kz = (float(t) for t in r.normal(size=3) * 6.0)
            v = v + torch.cos(kx * x + ky * y + kz * z + float(r.uniform(0, 2 * math.pi))) * float(r.normal())
        out[..., c] = v
    out += 0.02 * torch.randn(out.shape, generator=g, **f8)
    out /= out.norm(dim=-1, keepdim=True)
    return out.reshape(-1, 3)


def _Ms(mat, shape, seed):
    """Saturation magnetisation per cell (float), or the uniform value."""
    nx, ny, nz = shape
    if mat.get("disc"):
        x = (np.arange(nx) + 0.5) / nx * 2 - 1
        y = (np.arange(ny) + 0.5) / ny * 2 - 1
        inside = x[None, :] ** 2 + y[:, None] ** 2 <= 1.0
        return np.broadcast_to(np.where(inside, mat["Ms"], 0.0), (nz, ny, nx)).reshape(-1).copy()
    if mat.get("vary"):
        return np.random.default_rng(seed + 7919).uniform(0.86, 1.14, nx * ny * nz) * mat["Ms"]
    return mat["Ms"]


def _m0(case, shape, seed):
    m = _texture(shape, seed)
    Ms = _Ms(MATERIALS[case["material"]], shape, seed)
    if not np.isscalar(Ms):
        m[torch.from_numpy(Ms == 0).to(m.device)] = 0.0
    return m


def _cells(case):
    return tuple(case.get(k, 2.0) * 1e-9 for k in ("dx", "dy", "dz"))


# --------------------------------------------------------- the user's side --
_INTEGRATOR = {"rk4": "RungeKutta", "batch": "RungeKutta", "adjoint": "RungeKutta", "heun": "Heun",
               "dopri": "DormandPrince", "relax": None}


def _build(case, shape, seed):
    import mmcuda as mm

    mat = MATERIALS[case["material"]]
    mm.set_precision(np.float32 if case["form"] == "f32" else np.float64)
    dx, dy, dz = _cells(case)
    mesh = mm.FDMesh(nx=shape[0], ny=shape[1], nz=shape[2], dx=dx, dy=dy, dz=dz)
    integ = _INTEGRATOR[case["kind"]]
    if integ is None:
        sim = mm.Sim(mesh, driver="SD", save_data=False)
    else:
        sim = mm.Sim(mesh, driver="LLG", integrator=integ, save_data=False)
    sim.driver.alpha = mat["alpha"]
    sim.driver.gamma = GAMMA
    mm.set_Ms(sim, _Ms(mat, shape, seed))
    m0 = _m0(case, shape, seed).reshape(-1).cpu().numpy()
    mm.add_exch(sim, mat["A"])
    if "Dbulk" in mat:
        mm.add_dmi(sim, mat["Dbulk"], type="bulk")
    if "Dint" in mat:
        mm.add_dmi(sim, mat["Dint"], type="interfacial")
    if "Ku" in mat:
        mm.add_anis(sim, mat["Ku"], axis=(0, 0, 1))
    if "B" in mat:
        mm.add_zeeman(sim, tuple(b / MU0 for b in mat["B"]))
    if "sot" in mat:
        aj, bj, p = mat["sot"]
        mm.add_sot(sim, aj, bj, p)
    mm.add_demag(sim)
    sim.spin = m0
    return sim, m0


def prepare(case, seed):
    from mmcuda import _lib

    kind = case["kind"]
    dtype = torch.float32 if case["form"] == "f32" else torch.float64
    st = dict(case=case, sims=[], m0=[], out=[])
    for i, shape in enumerate(_shapes(case)):
        sim, m0 = _build(case, shape, seed + 1000 * i)
        st["sims"].append(sim)
        n3 = m0.size
        # page-locked host buffers, as a program that copies m every pass keeps
        st["out"].append(torch.empty(n3, dtype=dtype, pin_memory=True).numpy())
        if kind in ("dopri", "relax", "adjoint"):
            h = torch.empty(n3, dtype=torch.float64, pin_memory=True)
            h.copy_(torch.from_numpy(m0))
            st["m0"].append(h.numpy())
    if kind == "batch":
        st["batch"] = _lib.Batch([s._h for s in st["sims"]])
    if kind == "adjoint":
        st["target"] = _texture(_shapes(case)[0], seed + 17).reshape(-1).cpu().numpy()
    return st


def run(st):
    import mmcuda as mm
    from mmcuda import adjoint

    case = st["case"]
    kind, sim = case["kind"], st["sims"][0]
    if kind in ("rk4", "heun"):
        # one output interval of a longer run
        mm.run_rk4(sim, case["steps"], case["dt"])
    elif kind == "dopri":
        # a run from a given state over a time span
        sim.spin = st["m0"][0]
        sim._h.call("mm_dopri_reset")
        mm.run_until(sim, case["span"], save_data=False)
    elif kind == "relax":
        sim.spin = st["m0"][0]
        mm.relax(sim, max_steps=case["steps"], stopping_dmdt=0.0)
    elif kind == "batch":
        st["batch"].rk4_run(case["dt"], case["steps"])
        return {"m": [s._h.get_m(out=o) for s, o in zip(st["sims"], st["out"])]}
    elif kind == "adjoint":
        sim.spin = st["m0"][0]
        mT = adjoint.record(sim, case["steps"], case["dt"], case["every"])
        g = adjoint.backward(sim, 2 * (mT - st["target"]))
        return {"m": mT, "g_m0": g["m0"], "g_Ms": g["Ms"], "g_Ku": g["Ku"], "g_D": g["D"]}
    return {"m": sim._h.get_m(out=st["out"][0])}


# -------------------------------------------------------------------- work --
def _evals(case):
    """Right-hand-side evaluations of one pass (adaptive spans: a nominal step)."""
    if case["kind"] == "dopri":
        nominal = 5e-14 if case["material"] in ("chiral", "block", "interface") else 2e-13
        return 7 * max(1, round(case["span"] / nominal))
    per = {"rk4": 4, "batch": 4, "heun": 2, "relax": 1, "adjoint": 12}[case["kind"]]
    return per * case["steps"]


def work(case):
    """An evaluation reads the state, Ms and the demag tensor (six values a
    cell) and writes the next state; its convolution takes six real transforms
    of the doubled mesh and the 3 x 3 product, its local terms ~100 operations
    a cell."""
    w = 4 if case["form"] == "f32" else 8
    nbytes = flops = 0.0
    for nx, ny, nz in _shapes(case):
        n = nx * ny * nz
        padded = 1.0
        for d in (nx, ny, nz):
            padded *= 2 * d if d > 1 else 1
        nbytes += 13 * n * w * _evals(case) + 3 * n * w
        flops += (6 * 2.5 * padded * math.log2(max(2.0, padded)) + 15 * padded + 100 * n) * _evals(case)
    return {"bytes": nbytes, "flops": flops}


# --------------------------------------------------- the same in 64 bits ---
def _newell_f(x, y, z):
    """f of Newell, Williams and Dunlop (1993) in extended precision."""
    x2, y2, z2 = x * x, y * y, z * z
    R = np.sqrt(x2 + y2 + z2)
    with np.errstate(divide="ignore", invalid="ignore"):
        f = (2 * x2 - y2 - z2) * R / 6
        f = f - np.where(x2 > 0, x * y * z * np.arctan(y * z / (x * R)), 0)
        f = f + np.where(x2 + z2 > 0, y * (z2 - x2) / 2 * np.arcsinh(y / np.sqrt(x2 + z2)), 0)
        f = f + np.where(x2 + y2 > 0, z * (y2 - x2) / 2 * np.arcsinh(z / np.sqrt(x2 + y2)), 0)
    return np.where(R > 0, f, 0)


def _newell_g(x, y, z):
    x2, y2, z2 = x * x, y * y, z * z
    R = np.sqrt(x2 + y2 + z2)
    with np.errstate(divide="ignore", invalid="ignore"):
        g = -x * y * R / 3
        g = g - np.where(z2 > 0, z2 * z / 6 * np.arctan(x * y / (z * R)), 0)
        g = g - np.where(y2 > 0, y2 * z / 2 * np.arctan(x * z / (y * R)), 0)
        g = g - np.where(x2 > 0, x2 * z / 2 * np.arctan(y * z / (x * R)), 0)
        g = g + np.where(x2 + y2 > 0, x * y * z * np.arcsinh(z / np.sqrt(x2 + y2)), 0)
        g = g + np.where(y2 + z2 > 0, y * (3 * z2 - y2) / 6 * np.arcsinh(x / np.sqrt(y2 + z2)), 0)
        g = g + np.where(x2 + z2 > 0, x * (3 * z2 - x2) / 6 * np.arcsinh(y / np.sqrt(x2 + z2)), 0)
    return np.where(R > 0, g, 0)


def _tensor_spectrum(shape, cell):
    """Six demag tensor spectra on the doubled mesh (real part of rfftn of the
    tensor mirrored with its parities), near field within 60 cells, dipoles
    beyond."""
    nx, ny, nz = shape
    mx = max(cell)
    dx, dy, dz = (c / mx for c in cell)
    dev = "cuda"
    P = [2 * d if d > 1 else 1 for d in (nx, ny, nz)]
    perms = [("f", (0, 1, 2)), ("f", (1, 0, 2)), ("f", (2, 1, 0)), ("g", (0, 1, 2)), ("g", (0, 2, 1)), ("g", (1, 2, 0))]
    parity = [(0, 0, 0), (0, 0, 0), (0, 0, 0), (1, 1, 0), (1, 0, 1), (0, 1, 1)]
    ld = np.longdouble
    e = [min(n, int(60.0 / d) + 2) for n, d in zip((nx, ny, nz), (dx, dy, dz))]  # near-field offsets 0..e-1
    axes = [np.arange(-1, e[k] + 1).astype(ld) * ld((dx, dy, dz)[k]) for k in range(3)]
    X = np.broadcast_arrays(axes[0][None, None, :], axes[1][None, :, None], axes[2][:, None, None])
    i = torch.arange(nx, dtype=torch.float64, device=dev)[None, None, :] * dx
    j = torch.arange(ny, dtype=torch.float64, device=dev)[None, :, None] * dy
    k = torch.arange(nz, dtype=torch.float64, device=dev)[:, None, None] * dz
    far = torch.sqrt(i * i + j * j + k * k) > 60.0
    r2 = (i * i + j * j + k * k).clamp_min(1e-300)
    V4pi = dx * dy * dz / (4 * math.pi)
    co = (i, j, k)
    out = []
    for (fn, p), par in zip(perms, parity):
        F = (_newell_f if fn == "f" else _newell_g)(X[p[0]], X[p[1]], X[p[2]])
        for ax in range(3):  # second difference along each axis
            F = np.moveaxis(F, ax, 0)
            F = 2 * F[1:-1] - F[:-2] - F[2:]
            F = np.moveaxis(F, 0, ax)
        near = torch.from_numpy((F / (4 * ld(np.pi) * ld(dx) * ld(dy) * ld(dz))).astype(np.float64)).to(dev)
        if fn == "f":
            u, v, w = (co[q] for q in p)
            T = -(2 * u * u - v * v - w * w) / (r2 * r2 * torch.sqrt(r2)) * V4pi
        else:
            T = -3 * co[p[0]] * co[p[1]] / (r2 * r2 * torch.sqrt(r2)) * V4pi
        T = T.expand(nz, ny, nx).clone()
        T[:e[2], :e[1], :e[0]] = torch.where(far[:e[2], :e[1], :e[0]], T[:e[2], :e[1], :e[0]], near)
        for ax, (n, L) in enumerate(((nx, P[0]), (ny, P[1]), (nz, P[2]))):
            if n == 1:
                continue
            d = 2 - ax
            shp = list(T.shape)
            shp[d] = 1
            mir = torch.flip(T.narrow(d, 1, n - 1), (d,))
            T = torch.cat((T, torch.zeros(shp, dtype=T.dtype, device=dev), -mir if par[ax] else mir), d)
        S = torch.fft.rfftn(T, dim=(0, 1, 2))
        out.append(S.real.contiguous())
        del T, S
    return out, P


class _Exact:
    """Effective field and LLG right-hand side of a case in float64."""

    def __init__(self, case, shape, seed):
        self.mat = MATERIALS[case["material"]]
        self.shape = shape
        self.cell = _cells(case)
        nx, ny, nz = shape
        n = nx * ny * nz
        Ms = _Ms(self.mat, shape, seed)
        Ms = np.full(n, Ms) if np.isscalar(Ms) else Ms
        self.Ms = torch.from_numpy(Ms).to("cuda").reshape(nz, ny, nx)
        self.Ku = torch.full_like(self.Ms, self.mat.get("Ku", 0.0))
        self.D = torch.full_like(self.Ms, self.mat.get("Dint", 0.0))
        self.spec, self.P = _tensor_spectrum(shape, self.cell)
        self.m0 = _m0(case, shape, seed).T.reshape(3, nz, ny, nx).contiguous()

    def _demag(self, M):
        Px, Py, Pz = self.P
        nx, ny, nz = self.shape
        s = (Pz, Py, Px)
        xx, yy, zz, xy, xz, yz = self.spec
        F = [torch.fft.rfftn(M[c], s=s, dim=(0, 1, 2)) for c in range(3)]
        out = []
        for a, b, c in ((xx, xy, xz), (xy, yy, yz), (xz, yz, zz)):
            # component parities make every spectrum real
            out.append(-torch.fft.irfftn(F[0] * a + F[1] * b + F[2] * c, s=s, dim=(0, 1, 2))[:nz, :ny, :nx])
        return torch.stack(out)

    def field(self, m):
        mat = self.mat
        Ms = self.Ms
        mMs = Ms * MU0
        inv = torch.where(mMs > 0, 1.0 / torch.where(mMs > 0, mMs, torch.ones_like(mMs)), torch.zeros_like(mMs))
        dx = self.cell
        f = [torch.zeros_like(Ms) for _ in range(3)]
        A, Db = mat["A"], mat.get("Dbulk", 0.0)
        for ax in range(3):
            if self.shape[ax] == 1:
                continue
            d = 2 - ax
            n = self.shape[ax]
            for up in (0, 1):
                # value of the neighbour at -1 (up = 0) or +1 (up = 1), zero outside
                src = (lambda t: t.narrow(t.dim() - 3 + d, 1, n - 1)) if up else \
                      (lambda t: t.narrow(t.dim() - 3 + d, 0, n - 1))

                def shift(t):
                    pad = [0, 0, 0, 0, 0, 0]
                    pad[2 * ax + (1 if up else 0)] = 1
                    return torch.nn.functional.pad(src(t), pad)

                mn, Mn = shift(m), shift(Ms)
                on = (Mn > 0).to(Ms.dtype)
                c = 2 * A / dx[ax] ** 2 * on
                for q in range(3):
                    f[q] = f[q] + c * (mn[q] - m[q])
                sgn = 1.0 if up else -1.0
                if Db:
                    # sum of (D/d) r x m_neighbour, r = -+ e_ax towards the neighbour
                    e = [0.0, 0.0, 0.0]
                    e[ax] = -sgn
                    w = Db / dx[ax] * on
                    f[0] = f[0] + w * (e[1] * mn[2] - e[2] * mn[1])
                    f[1] = f[1] + w * (e[2] * mn[0] - e[0] * mn[2])
                    f[2] = f[2] + w * (e[0] * mn[1] - e[1] * mn[0])
                if "Dint" in mat and ax < 2:
                    Dn = shift(self.D)
                    w = torch.where(on > 0, 2 * self.D * Dn / (self.D + Dn), torch.zeros_like(Dn)) / dx[ax]
                    # r = +y, -y, -x, +x for the neighbours at -x, +x, -y, +y
                    e = (0.0, -sgn, 0.0) if ax == 0 else (sgn, 0.0, 0.0)
                    f[0] = f[0] + w * (e[1] * mn[2] - e[2] * mn[1])
                    f[1] = f[1] + w * (e[2] * mn[0] - e[0] * mn[2])
                    f[2] = f[2] + w * (e[0] * mn[1] - e[1] * mn[0])
        h = torch.stack(f) * inv
        if "Ku" in mat:
            h = h + torch.stack((torch.zeros_like(Ms), torch.zeros_like(Ms), 2 * self.Ku * m[2] * inv))
        h = h + self._demag(Ms * m)
        if "B" in mat:
            h = h + torch.tensor(mat["B"], dtype=m.dtype, device=m.device).reshape(3, 1, 1, 1) / MU0
        if "sot" in mat:
            aj, bj, p = mat["sot"]
            p = torch.tensor(p, dtype=m.dtype, device=m.device).reshape(3, 1, 1, 1).expand_as(m)
            h = h + aj / GAMMA * torch.linalg.cross(m, p, dim=0) + bj / GAMMA * p
        return h

    def rhs(self, m):
        h = self.field(m)
        al = self.mat["alpha"]
        hp = (m * m).sum(0) * h - (m * h).sum(0) * m
        return -GAMMA / (1 + al * al) * (torch.linalg.cross(m, hp, dim=0) - al * hp)

    @staticmethod
    def unit(m):
        n = (m * m).sum(0)
        return m / torch.sqrt(torch.where(n > 0, n, torch.ones_like(n)))

    def rk4(self, m, h):
        k1 = self.rhs(m)
        k2 = self.rhs(m + 0.5 * h * k1)
        k3 = self.rhs(m + 0.5 * h * k2)
        k4 = self.rhs(m + h * k3)
        return self.unit(m + h / 6 * (k1 + 2 * k2 + 2 * k3 + k4))

    def heun(self, m, h):
        k1 = self.rhs(m)
        k2 = self.rhs(m + h * k1)
        return self.unit(m + 0.5 * h * (k1 + k2))

    def dopri(self, m, span, tol=1e-6):
        a = [[1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9],
             [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
             [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656],
             [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]]
        w = [71 / 57600, 0, -71 / 16695, 71 / 1920, -17253 / 339200, 22 / 525, -1 / 40]
        r = float(self.rhs(m).abs().max()) / (0.824 * tol ** 0.2)
        step = min(1e-12, 0.001 / r if 1e-12 * r > 0.001 else 1e-12)
        # a fresh integrator takes its first step at the estimate, unclipped
        t = 0.0
        while t < span:
            k = []
            y = m
            for s in range(7):
                k.append(self.rhs(y))
                if s < 6:
                    y = m
                    for c, kk in zip(a[s], k):
                        if c:
                            y = y + (c * step) * kk
                    if s == 5:
                        y = self.unit(y)
            err = sum(c * kk for c, kk in zip(w, k) if c)
            err = float((err / (1 + y.abs())).abs().max()) * step / tol
            if err <= 1.0:
                t += step
                m = y
                step *= min(5.0, max(0.2, 0.824 * (1 / err) ** 0.2))
                if t < span and t + step > span:
                    step = span - t
            else:
                step *= min(5.0, max(0.2, 0.824 * (1 / err) ** 0.25))
        return m

    def descend(self, m, steps):
        pre = gk = None
        for s in range(steps):
            h = self.field(m)
            f = torch.linalg.cross(m, h, dim=0)
            g = torch.linalg.cross(m, f, dim=0)
            if s == 0:
                tau = 1e-10
            else:
                ds, dg = m - pre, g - gk
                s1, s2, s3 = float((ds * ds).sum()), float((ds * dg).sum()), float((dg * dg).sum())
                tau = abs(s2 / s3 if s3 else 1e-10) if s % 2 == 0 else abs(s1 / s2 if s2 else 1e-10)
                tau = min(tau, 1.0)
            pre, gk = m, g
            q = 0.25 * (f * f).sum(0) * tau * tau
            m = ((1 - q) * m - tau * g) / (1 + q)
            if (s + 1) % 10 == 0:
                m = self.unit(m)
        return m


def _aos(m):
    return m.reshape(3, -1).T.contiguous().reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    shapes = _shapes(case)
    if kind == "adjoint":
        ex = _Exact(case, shapes[0], seed)
        m0 = ex.m0.clone().requires_grad_(True)
        for t in (ex.Ms, ex.Ku, ex.D):
            t.requires_grad_(True)
        from torch.utils.checkpoint import checkpoint

        m = m0
        for _ in range(case["steps"]):
            m = checkpoint(ex.rk4, m, case["dt"], use_reentrant=False)
        target = _texture(shapes[0], seed + 17).T.reshape(m.shape)
        ((m - target) ** 2).sum().backward()
        return {"m": _aos(m.detach()), "g_m0": _aos(m0.grad), "g_Ms": ex.Ms.grad.reshape(-1),
                "g_Ku": ex.Ku.grad.reshape(-1), "g_D": ex.D.grad.reshape(-1)}
    out = []
    with torch.no_grad():
        for i, shape in enumerate(shapes):
            ex = _Exact(case, shape, seed + 1000 * i)
            m = ex.m0
            if kind == "dopri":
                m = ex.dopri(m, case["span"])
            elif kind == "relax":
                m = ex.descend(m, case["steps"])
            else:
                step = ex.heun if kind == "heun" else ex.rk4
                for _ in range(case["steps"]):
                    m = step(m, case["dt"])
            out.append(_aos(m))
    return {"m": out if kind == "batch" else out[0]}
