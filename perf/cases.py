"""Workloads by which the speed of this framework is measured.

Each case is one pass of what a user's program does with the library through
its Python entry points (fdtd_b200.grid, fdtd_b200.problem): advance a grid, a
batch of grids or an adjoint gradient, and have the new state (every E and H
component, on the device, by copy_plane) and the spectra in hand afterwards.

  listed()            the cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) the inputs and handles such a program holds
  run(state)          one pass, returning its outputs
  work(case)          the bytes and operations a pass cannot do without
  exact(case, seed)   the same outputs in 64 bits by plain torch
"""
import math

import numpy as np
import torch

EPS0, MU0, C0 = 8.854e-12, 4.0e-7 * math.pi, 2.99792458e8
ETA = math.sqrt(MU0 / EPS0)
DX = 1e-6
TE, TM, THREED = 1, 2, 3
MODES = {"TE": TE, "TM": TM, "3D": THREED}


def listed():
    grid = dict(kind="grid", mode="TM", prec="f32", nx=256, ny=256, nz=1, npml=16, material="vacuum", tfsf=False, dft="none", nfreq=3, steps=1)
    cases = [
        # a program that couples something of its own to every step: a small 2D grid, one step per call
        dict(grid, name="te160x96_f32_step1", mode="TE", nx=160, ny=96, npml=10, material="rects"),
        # the plain FP64 method at its usual size: a vacuum grid, point source, spectra along a row, a whole run
        dict(grid, name="tm256_f64_run", prec="f64", dft="row", steps=2000),
        # the same kind of run in FP32, odd extents, dielectric objects
        dict(grid, name="tm317x233_f32_run", nx=317, ny=233, npml=12, material="rects", dft="row", steps=1000),
        # a 2D scattering run in FP64: a plane wave on a Drude disk
        dict(grid, name="te600x450_f64_drude", mode="TE", prec="f64", nx=600, ny=450, npml=12, material="drude", tfsf=True, dft="row", steps=200),
        # a large 2D FP32 grid, beyond the caches
        dict(grid, name="te3001x2047_f32", mode="TE", nx=3001, ny=2047, npml=12, material="rects", dft="row", steps=100),
        # many independent 2D grids of uneven sizes advanced together, tuned
        dict(kind="batch", name="batch64_te_f32", mode="TE", problems=64, nmin=128, nmax=1024, npml=10, steps=240),
        # one gradient of an inverse design: forward and backward, as each iteration of an optimiser asks for
        dict(kind="adjoint", name="adjoint512_f32", nx=512, ny=512, npml=16, design=128, steps=4000, ckpt=64),
        # 3D grids: a sphere in a plane-wave box with spectra on the faces of a box around it, small to large
        dict(grid, name="drude132x64x60_f32", mode="3D", nx=132, ny=64, nz=60, npml=12, material="drude", tfsf=True, dft="faces", nfreq=8, steps=500),
        dict(grid, name="drude173x150x141_f64", mode="3D", prec="f64", nx=173, ny=150, nz=141, npml=12, material="drude", tfsf=True, dft="faces", nfreq=4, steps=100),
        dict(grid, name="drude384_f32", mode="3D", nx=384, ny=384, nz=384, npml=12, material="drude", tfsf=True, dft="faces", nfreq=8, steps=256),
        # dispersive media everywhere, spectra on the central plane
        dict(grid, name="lorentz260x200x161_f64", mode="3D", prec="f64", nx=260, ny=200, nz=161, npml=16, material="lorentz2", dft="plane", nfreq=4, steps=40),
        dict(grid, name="lorentz768_f32", mode="3D", nx=768, ny=768, nz=768, npml=16, material="lorentz2", dft="plane", nfreq=4, steps=24),
    ]
    return cases


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    pick = rng.random()
    if pick < 0.12:
        nmin = _log(rng, 64, 256)
        return dict(kind="batch", mode=rng.choice(["TE", "TM"]), problems=_log(rng, 4, 64), nmin=nmin, nmax=nmin * rng.choice([2, 4]), npml=rng.choice([8, 10, 12]),
                    steps=_log(rng, 20, 400))
    if pick < 0.24:
        npml = rng.choice([8, 12, 16])
        nx, ny = _log(rng, 160, 700), _log(rng, 160, 700)
        return dict(kind="adjoint", nx=nx, ny=ny, npml=npml, design=_log(rng, 24, (min(nx, ny) - 2 * npml) // 2 - 16), steps=_log(rng, 300, 4000), ckpt=rng.choice([32, 50, 64]))
    prec = rng.choice(["f32", "f32", "f64"])
    npml = rng.choice([8, 10, 12, 16])
    if pick < 0.66:
        mode = rng.choice(["TE", "TM"])
        nx, ny, nz = _log(rng, 64, 3000), _log(rng, 64, 3000), 1
        steps = max(1, min(_log(rng, 1, 2000), int(1e9 // (nx * ny))))
        material = rng.choice(["vacuum", "rects", "rects", "drude", "lorentz1"])
        dft = rng.choice(["none", "row"])
    else:
        mode = "3D"
        lo, hi = 2 * npml + 20, 400 if prec == "f32" else 260
        nx, ny, nz = (_log(rng, lo, hi) for _ in range(3))
        steps = max(1, min(_log(rng, 20, 1000), int((4e9 if prec == "f32" else 1e9) // (nx * ny * nz))))
        material = rng.choice(["vacuum", "rects", "drude", "lorentz1", "lorentz2"])
        dft = rng.choice(["none", "plane", "faces"])
    roomy = min(nx, ny, nz if mode == "3D" else ny) >= 2 * (npml + 8) + 8
    tfsf = roomy and not material.startswith("lorentz") and rng.random() < 0.4
    if dft == "faces" and not roomy:
        dft = "plane"
    return dict(kind="grid", mode=mode, prec=prec, nx=nx, ny=ny, nz=nz, npml=npml, material=material, tfsf=tfsf, dft=dft, nfreq=rng.choice([1, 3, 4, 8]), steps=steps)


# ---------------------------------------------------------------- inputs, as plain arrays

def _e_comps(mode):
    return {TE: [0, 1], TM: [2], THREED: [0, 1, 2]}[mode]


def _h_comps(mode):
    return {TE: [2], TM: [0, 1], THREED: [0, 1, 2]}[mode]


def _dt(mode):
    return 0.98 / math.sqrt(3.0 if mode == THREED else 2.0) * DX / C0


def _pulse(n, t0=60.0, spread=20.0, offset=0.0):
    return np.exp(-(((np.arange(n) + offset - t0) / spread) ** 2))


def _boxes(rng, shape, npml, count, mats, ids):
    """`count` axis-aligned dielectric boxes of 8 to 64 cells a side outside the CPML."""
    lo = npml + 2
    for _ in range(count):
        sl = []
        for n in shape:
            if n == 1:
                sl.append(slice(0, 1))
                continue
            w = max(1, min(int(rng.integers(8, 65)), n - 2 * lo - 1))
            x0 = int(rng.integers(lo, max(lo + 1, n - lo - w)))
            sl.append(slice(x0, x0 + w))
        mats.append(("const", float(rng.uniform(1.0, 12.0)), []))
        ids[sl[2], sl[1], sl[0]] = len(mats) - 1


def _inputs(case, seed):
    """Everything a grid's run depends on, from the seed alone: materials as
    (kind, eps_inf, poles in grid units), sources, plane wave, DFT boxes."""
    mode, shape = MODES[case["mode"]], (case["nx"], case["ny"], case["nz"])
    nx, ny, nz = shape
    dim = 3 if mode == THREED else 2
    rng = np.random.default_rng([int(seed), nx, ny, nz])
    npml, steps, dt = case["npml"], case["steps"], _dt(mode)
    mats, ids, blocks = [("vacuum", 1.0, [])], None, None
    kind = case["material"]
    if kind == "rects":
        ids = np.zeros((nz, ny, nx), np.uint8)
        _boxes(rng, shape, npml, 10, mats, ids)
    elif kind == "drude":
        wp, gam = 0.3 / dt * float(rng.uniform(0.8, 1.0)), 0.01 / dt
        mats.append(("drude", 1.0, [(1.0, wp, gam)]))
        r = min(shape[:dim]) // 6
        ax = [np.arange(n) - n // 2 for n in shape]
        ids = ((ax[2][:, None, None] ** 2 if dim == 3 else np.zeros((1, 1, 1), int)) + ax[1][None, :, None] ** 2 + ax[0][None, None, :] ** 2 <= r * r).astype(np.uint8)
    elif kind.startswith("lorentz"):
        # the poles everywhere, eps_inf by blocks of 32 cells a side
        poles = [(1.5, 0.1 / dt, 0.005 / dt), (0.8, 0.25 / dt, 0.02 / dt)][: int(kind[-1])]
        nb = [(n + 31) // 32 for n in shape]
        eps = rng.uniform(1.0, 6.0, size=nb[0] * nb[1] * nb[2])
        mats = [("lorentz", float(e), poles) for e in eps]
        blocks = np.arange(eps.size, dtype=np.uint16).reshape(nb[2], nb[1], nb[0])
    tfsf = None
    if case["tfsf"]:
        inset = npml + 6
        tfsf = dict(lo=[inset] * dim, hi=[n - 1 - inset for n in shape[:dim]], origin=[float(n // 2) for n in shape], k=(1.0, 0.0, 0.0), aux=max(shape),
                    vals=float(rng.uniform(0.5, 2.0)) * _pulse(steps, offset=1.0),
                    pol_e=(0.0, -1.0, 0.0) if mode == TE else (0.0, 0.0, 1.0), pol_h=(0.0, 0.0, 1.0) if mode == TE else (0.0, 1.0, 0.0))
    src = None
    if tfsf is None:
        pos = tuple(int(rng.integers(npml + 2, n - npml - 2)) if n > 1 else 0 for n in shape)
        amp = float(rng.uniform(0.5, 2.0))
        src = dict(comp=2, pos=pos, target="H" if mode == TE else "E", vals=amp * _pulse(steps) / (ETA if mode == TE else 1.0))
    freqs = [0.01 * (q + 1) for q in range(case["nfreq"])]
    e0 = {TE: 1, TM: 2, THREED: 2}[mode]
    dfts = []
    if case["dft"] == "row":
        dfts.append((e0, (0, ny // 2, 0), (nx - 1, ny // 2, 0)))
    elif case["dft"] == "plane":
        dfts.append((e0, (0, 0, nz // 2), (nx - 1, ny - 1, nz // 2)))
    elif case["dft"] == "faces":
        a0 = npml + 3
        for a in range(3):
            for side in (0, 1):
                lo, hi = [a0] * 3, [n - 1 - a0 for n in shape]
                lo[a] = hi[a] = a0 if side == 0 else shape[a] - 1 - a0
                for b in range(3):
                    if b != a:
                        dfts += [(b, tuple(lo), tuple(hi)), (3 + b, tuple(lo), tuple(hi))]
    return dict(mode=mode, shape=shape, dim=dim, dt=dt, npml=npml, steps=steps, mats=mats, ids=ids, blocks=blocks, tfsf=tfsf, src=src, freqs=freqs, dfts=dfts, f32=case["prec"] == "f32")


def _waves(inp, seed, component, half):
    """The starting value of one component (half 0: E, 1: eta * H): a few smooth
    waves with wavelengths of 12 to 90 cells, zero on the fixed outer ring, in
    the precision the grid holds."""
    g = np.random.default_rng([int(seed), 77, component, half])
    nx, ny, nz = inp["shape"]
    out = torch.zeros((nz, ny, nx), dtype=torch.float32 if inp["f32"] else torch.float64, device="cuda")
    fac = []
    for n in (nz, ny, nx):
        x = np.arange(n)[None, :]
        w = np.sin(2 * np.pi * x / g.uniform(12, 90, size=(3, 1)) + g.uniform(0, 6.3, size=(3, 1))) if n > 1 else np.ones((3, 1))
        if n > 1:
            w[:, 0] = w[:, -1] = 0.0
        fac.append(torch.tensor(w, dtype=out.dtype, device="cuda"))
    for m in range(3):
        out.addcmul_((fac[0][m][:, None] * fac[1][m][None, :])[:, :, None], fac[2][m][None, None, :], value=float(g.uniform(0.2, 1.0)))
    return out


def _problem(inp, P):
    p = P.Problem(inp["mode"], inp["shape"], DX, inp["dt"])
    for a in range(inp["dim"]):
        for s in (0, 1):
            p.pml[(a, s)] = inp["npml"]
    make = {"vacuum": lambda e, q: P.Material.vacuum(), "const": lambda e, q: P.Material.constant(e), "drude": lambda e, q: P.Material.drude(e, *q[0][1:]),
            "lorentz": lambda e, q: P.Material.lorentz(e, q)}
    p.materials = [make[k](e, q) for k, e, q in inp["mats"]]
    p.ids = inp["ids"]
    if inp["blocks"] is not None:
        p.block_ids, p.block_shift = inp["blocks"], 5
    if inp["src"]:
        p.sources.append(P.Source(inp["src"]["comp"], inp["src"]["pos"], inp["src"]["vals"], inp["src"]["target"]))
    if inp["tfsf"]:
        t = inp["tfsf"]
        p.tfsf = P.TFSF(t["aux"], t["vals"], tuple(t["origin"]), t["k"], t["pol_e"], t["pol_h"], P.tfsf_box_planes(inp["mode"], t["lo"], t["hi"]))
    for comp, lo, hi in inp["dfts"]:
        p.dfts.append(P.DFTRegion(comp, lo, hi, inp["freqs"]))
    p.steps = inp["steps"]
    return p


def _load(g, inp, seed):
    """A grid whose fields hold _waves, as after reading back a saved run."""
    for half, comps in ((0, _e_comps(inp["mode"])), (1, _h_comps(inp["mode"]))):
        for c in comps:
            w = _waves(inp, seed, c, half)
            if half == 1 and not inp["f32"]:
                w /= ETA
            torch.cuda.synchronize()
            for k in range(inp["shape"][2]):
                g.copy_plane("EH"[half] + "xyz"[c], k, w[k].data_ptr(), True)
            if half == 0 and not inp["f32"] and inp["blocks"] is not None:
                w *= EPS0 * _eps(inp)
                g.set("D" + "xyz"[c], w.cpu().numpy())
            g.synchronize()
    if not inp["f32"]:
        if inp["blocks"] is None:
            g.material_explicit(0)
        g.material_explicit(1)
    g.synchronize()


def _config3(case, seed):
    """The grids of a batch: extents uniform in [nmin, nmax], ten dielectric
    rectangles and a point source each."""
    rng = np.random.default_rng(case["nmin"] * 1000 + case["problems"])  # the sizes are the case's, not the seed's
    sizes = rng.integers(case["nmin"], case["nmax"] + 1, size=(case["problems"], 2))
    one = dict(mode=case["mode"], prec="f32", nz=1, npml=case["npml"], material="rects", tfsf=False, dft="none", nfreq=1, steps=case["steps"])
    return [dict(one, nx=int(a), ny=int(b)) for a, b in sizes]


def _design(case, seed):
    """The permittivity, source values and boxes of one gradient."""
    rng = np.random.default_rng([int(seed), 4])
    nx, ny, d = case["nx"], case["ny"], case["design"]
    x0, y0 = (nx - d) // 2, (ny - d) // 2
    eps = np.zeros((1, ny, nx))
    eps[0, y0:y0 + d, x0:x0 + d] = rng.uniform(1.0, 12.0, size=(d, d))
    freq, n = 0.05, np.arange(case["steps"])
    vals = np.tanh(n * freq / 2.5) * np.sin(2 * np.pi * freq * n)
    col, pc, j0 = case["npml"] + 4, nx - 1 - (case["npml"] + 4), ny // 2 - 8
    return dict(eps=eps, vals=vals, freq=freq, col=col, probe=((pc, j0, 0), (pc, j0 + 15, 0)), design=((x0, y0, 0), (x0 + d - 1, y0 + d - 1, 0)))


# ---------------------------------------------------------------- a pass

class _GridRun:
    """A grid, the spectra it gathers and device arrays for its fields."""

    def __init__(self, case, seed):
        from fdtd_b200 import problem as P
        from fdtd_b200.grid import Grid
        inp = _inputs(case, seed)
        self.steps, self.f32, self.shape = inp["steps"], inp["f32"], inp["shape"]
        self.g = Grid.from_problem(_problem(inp, P), case["prec"])
        _load(self.g, inp, seed)
        self.g.prepare()
        nx, ny, nz = self.shape
        dtype = torch.float32 if self.f32 else torch.float64
        names = ["E" + "xyz"[c] for c in _e_comps(inp["mode"])] + ["H" + "xyz"[c] for c in _h_comps(inp["mode"])]
        self.out = {n: torch.empty((nz, ny, nx), dtype=dtype, device="cuda") for n in names}
        self.plane = nx * ny * self.out[names[0]].element_size()

    def fields(self):
        for name, t in self.out.items():
            for k in range(self.shape[2]):
                self.g.copy_plane(name, k, t.data_ptr() + k * self.plane, False)

    def run(self):
        self.g.step(self.steps)
        self.fields()
        out = dict(self.out)
        for q, h in enumerate(self.g.dft_handles):
            x = torch.from_numpy(self.g.dft(h))
            out["dft%d" % q] = x.to(torch.complex64) if self.f32 else x
        return out


class _BatchRun:
    """A tuned batch; the fields of all its grids one after another."""

    def __init__(self, case, seed):
        from fdtd_b200 import problem as P
        from fdtd_b200.grid import Batch, Grid
        self.steps, self.grids = case["steps"], []
        for q, c in enumerate(_config3(case, seed)):
            inp = _inputs(c, seed + 7919 * (q + 1))
            g = Grid.from_problem(_problem(inp, P), "f32")
            _load(g, inp, seed + 7919 * (q + 1))
            self.grids.append(g)
        self.batch = Batch(self.grids)
        self.batch.tune(8)
        mode = MODES[case["mode"]]
        total = sum(g.shape[0] * g.shape[1] for g in self.grids)
        self.out = {n: torch.empty(total, dtype=torch.float32, device="cuda") for n in ["E" + "xyz"[c] for c in _e_comps(mode)] + ["H" + "xyz"[c] for c in _h_comps(mode)]}

    def run(self):
        self.batch.step(self.steps)
        for name, t in self.out.items():
            at = t.data_ptr()
            for g in self.grids:
                g.copy_plane(name, 0, at, False)
                at += 4 * g.shape[0] * g.shape[1]
        return dict(self.out)


class _AdjointRun:
    """One iteration of an inverse design: the grid of the permittivity in
    hand, its objective and its gradient."""

    def __init__(self, case, seed):
        from fdtd_b200 import problem as P
        d = self.d = _design(case, seed)
        self.case = case
        p = self.p = P.Problem(TM, (case["nx"], case["ny"], 1), DX, _dt(TM))
        for a in (0, 1):
            for s in (0, 1):
                p.pml[(a, s)] = case["npml"]
        p.eps_map = d["eps"]
        p.sources.append(P.Source(2, (d["col"], 1, 0), d["vals"], "E", hi=(d["col"], case["ny"] - 2, 0)))
        p.steps = case["steps"]

    def run(self):
        from fdtd_b200.grid import Adjoint, Grid
        d = self.d
        g = Grid.from_problem(self.p, "f32")
        adj = Adjoint(g, *d["probe"], d["freq"], *d["design"], self.case["ckpt"])
        J = adj.forward(self.case["steps"])
        grad = adj.backward()
        adj.close()
        g.close()
        return {"J": np.float32(J), "grad": grad.astype(np.float32)}


def prepare(case, seed):
    return {"grid": _GridRun, "batch": _BatchRun, "adjoint": _AdjointRun}[case["kind"]](case, seed)


def run(state):
    return state.run()


# ---------------------------------------------------------------- what a pass cannot do without

def _step_work(case):
    """Bytes and operations of one step: every stored word that a step changes
    read and written once, ids read once, CPML integrators over their slabs,
    polarisation over its cells. FP64 stores D and B besides E and H."""
    mode, w = MODES[case["mode"]], 4 if case["prec"] == "f32" else 8
    n = [case["nx"] - 2, case["ny"] - 2] + ([case["nz"] - 2] if mode == THREED else [])
    cells = math.prod(n)
    ne, nh = len(_e_comps(mode)), len(_h_comps(mode))
    words = (ne + nh) * (2 if w == 4 else 3)
    slab = sum(min(2 * case["npml"] + 2, n[a]) * (cells // n[a]) for a in range(len(n)))
    pole_cells, pole_words = 0, 0
    if case["material"] == "drude":
        r = min(n) // 6
        pole_cells, pole_words = (4.19 * r ** 3 if mode == THREED else 3.14 * r * r), 2 if w == 4 else 4
    elif case["material"].startswith("lorentz"):
        pole_cells, pole_words = cells, 4 * int(case["material"][-1])
    byte = cells * words * w + slab * 2 * 2 * 2 * w + pole_cells * ne * pole_words * w + (cells if case["material"] in ("rects", "drude") else 0)
    flop = cells * (ne + nh) * (8 if mode == THREED else 5) + slab * 16 + pole_cells * ne * 3 * pole_words
    return float(byte), float(flop)


def work(case):
    if case["kind"] == "adjoint":
        # the forward's state once per step; the backward steps the forward
        # again and the adjoint state once
        one = dict(case, mode="TM", prec="f32", nz=1, material="rects")
        b, f = _step_work(one)
        return {"bytes": 3 * b * case["steps"] + 4 * case["design"] ** 2 * 4 * case["steps"], "flops": 3 * f * case["steps"]}
    grids = _config3(case, 0) if case["kind"] == "batch" else [case]
    byte = flop = 0.0
    for c in grids:
        b, f = _step_work(c)
        mode, w = MODES[c["mode"]], 4 if c["prec"] == "f32" else 8
        byte += b * c["steps"] + 2 * w * (len(_e_comps(mode)) + len(_h_comps(mode))) * c["nx"] * c["ny"] * c["nz"]
        flop += f * c["steps"]
    return {"bytes": byte, "flops": flop}


# ---------------------------------------------------------------- the same in 64 bits

def _grading(n, np_, dt, dx):
    """CPML coefficients of one axis, E and H, with CPML of np_ cells on both
    sides: convolutional PML graded with m = 3, m_a = 1, sigma_max =
    3.2 / (eta dx), kappa_max = 5, alpha_max = 0.05."""
    out = []
    for half in (0, 1):
        B, C, F, G = np.zeros(n), np.zeros(n), np.ones(n), np.zeros(n)
        for i in range(1, np_ + 2):
            x = (np_ - i + 1) / np_ - (0.5 / np_ if half else 0.0)
            inside = 0.0 <= x <= 1.0
            K = 1.0 + x ** 3 * 4.0 if inside else 1.0
            S = x ** 3 * 3.2 / (ETA * dx) if inside else 0.0
            A = (1.0 - x) * 0.05 if inside else 0.0
            nu = (S / K + A) / EPS0
            if nu == 0.0:
                b, c, f, g = 1.0, 0.0, 1.0 / K, 0.0
            else:
                b = math.exp(-dt * nu)
                c = S / K / (S + K * A) * (b - 1.0)
                u = -S / (EPS0 * K * K)
                f = 1.0 / K - (1.0 - b - nu * dt) * u / (nu * nu) / dt
                g = (1.0 - b) / nu / dt
            for at in (i, n - 1 - i if half else n - i):
                B[at], C[at], F[at], G[at] = b, c, f, g
        out.append((B, C, F, G))
    return out


def _aux(t, dt, steps):
    """Ez and Hy of the plane wave's 1D grid after each step."""
    L = t["aux"] + 50
    (eB, eC, eF, eG), (hB, hC, hF, hG) = _grading(L, 15, dt, DX)
    E, H, pe, ph = (np.zeros(L) for _ in range(4))
    Et, Ht = np.zeros((steps + 1, L)), np.zeros((steps + 1, L))
    last = 0.0
    for s in range(1, steps + 1):
        diff = H - np.concatenate(([0.0], H[:-1]))
        E[20] -= last
        E = E + dt / EPS0 * (eF / DX * diff + pe * eG)
        pe = eB * pe + eC / DX * diff
        last = t["vals"][s - 1] if s <= len(t["vals"]) else 0.0
        E[20] += last
        diff = np.concatenate((E[1:], [0.0])) - E
        H = H + dt / MU0 * (hF / DX * diff - ph * hG)
        ph = hB * ph - hC / DX * diff
        Et[s], Ht[s] = E, H
    return Et, Ht


def _eps(inp):
    e = torch.tensor([m[1] for m in inp["mats"]], dtype=torch.float64, device="cuda")
    if inp["ids"] is not None:
        return e[torch.as_tensor(inp["ids"], device="cuda").long()]
    if inp["blocks"] is None:
        return e[0].reshape(1, 1, 1)
    nx, ny, nz = inp["shape"]
    t = torch.as_tensor(inp["blocks"].astype(np.int64), device="cuda")
    at = [torch.arange(n, device="cuda") >> 5 for n in (nz, ny, nx)]
    return e[t[at[0]][:, at[1]][:, :, at[2]]]


def _levi(i, j, k):
    return (i - j) * (j - k) * (k - i) // 2


class _Exact:
    """The leapfrog update of E and eta * H with CPML, poles, a plane wave box
    and running spectra, in float64 by torch; 2D grids hold one plane."""

    def __init__(self, inp, seed):
        self.inp = inp
        mode, dim, dt = inp["mode"], inp["dim"], inp["dt"]
        nx, ny, nz = inp["shape"]
        self.comps = (_e_comps(mode), _h_comps(mode))
        self.F = [[_waves(inp, seed, c, h).double() if c in self.comps[h] else None for c in range(3)] for h in (0, 1)]
        self.inner = tuple(slice(1, n - 1) if n > 1 else slice(0, 1) for n in (nz, ny, nx))
        self.coef = [dt / (EPS0 * ETA * DX), ETA * dt / (MU0 * DX)]
        self.prof = [_grading(n, inp["npml"], dt, DX) if a < dim else None for a, n in enumerate(inp["shape"])]
        self.ie = 1.0 / _eps(inp)[self.inner] if inp["ids"] is not None or inp["blocks"] is not None else 1.0 / inp["mats"][0][1]
        self.poles = []
        rows = [m for m in inp["mats"] if m[2]]
        mask = 1.0
        if rows and inp["ids"] is not None:
            mask = (torch.as_tensor(inp["ids"], device="cuda") == 1).double()[self.inner]
        if rows:
            kind, _, poles = rows[0]
            for de, w, g in poles:
                if kind == "drude":
                    b = g * dt * 0.5
                    a_, b_, c_ = (1 - b) / (1 + b), (w * dt) ** 2, None
                else:
                    a_, b_, c_ = (1 - g * dt) / (1 + g * dt), (w * dt) ** 2 * de / (1 + g * dt), (w * dt) ** 2 / (1 + g * dt)
                one = dict(a=a_, b=b_ * mask, c=c_, J={}, P={})
                for c in self.comps[0]:
                    e = self.F[0][c][self.inner]
                    # the FP64 grid's starting current, as its explicit material update sets it
                    one["J"][c] = -((w * dt) ** 2) * mask * e / (1 + g * dt) if kind == "drude" and not inp["f32"] else torch.zeros_like(e)
                    one["P"][c] = torch.zeros_like(e) if kind != "drude" else None
                self.poles.append(one)
        # CPML integrators: (slice of the inner cells, B, C, G, psi) per half, component and axis
        self.slabs = [{}, {}]
        for h in (0, 1):
            for I in self.comps[h]:
                for J in range(dim):
                    if I == J:
                        continue
                    B, C, _, G = self.prof[J][h]
                    n = inp["shape"][J]
                    parts = []
                    for lo, hi in ((1, inp["npml"] + 2), (n - 2 - inp["npml"], n - 1)):
                        sl = [slice(None)] * 3
                        sl[2 - J] = slice(lo - 1, hi - 1)
                        col = [self._axis(v[lo:hi], J) for v in (B, self.coef[h] * C, G)]
                        parts.append([tuple(sl), *col, torch.zeros_like(self.F[h][I][self.inner][tuple(sl)])])
                    self.slabs[h][I, J] = parts
        self.scale = [[self._axis(self.coef[h] * self.prof[a][h][2][1:-1], a) if a < dim else None for a in range(3)] for h in (0, 1)]
        self.spectra = [torch.zeros((len(inp["freqs"]), *[h - l + 1 for l, h in zip(lo[::-1], hi[::-1])]), dtype=torch.complex128, device="cuda") for _, lo, hi in inp["dfts"]]
        self.last = 0.0
        self.planes = [[], []]
        if inp["tfsf"]:
            self.tabs = [torch.tensor(x, device="cuda") for x in _aux(inp["tfsf"], dt, inp["steps"])]
            self._plan_planes()

    @staticmethod
    def _axis(v, a):
        s = [1, 1, 1]
        s[2 - a] = -1
        return torch.tensor(np.ascontiguousarray(v), device="cuda").reshape(s)

    def _plan_planes(self):
        t, dim, shape = self.inp["tfsf"], self.inp["dim"], self.inp["shape"]
        L = t["aux"] + 50
        for A in range(dim):
            for side in (0, 1):
                lo, hi = list(t["lo"]) + [0] * (3 - dim), list(t["hi"]) + [0] * (3 - dim)
                lo[A] = hi[A] = t["lo"][A] - 1 if side == 0 else t["hi"][A]
                normal = 1.0 if side == 1 else -1.0
                for h in (0, 1):
                    for I in self.comps[h]:
                        K = 3 - I - A
                        if I == A or K not in self.comps[1 - h]:
                            continue
                        nd = L / 2.0 - (0.5 if h == 0 else 0.0)
                        off = (-0.5 if 0 == K else 0.0) if h == 0 else (0.0 if 0 == K else -0.5)
                        nd = nd + (np.arange(lo[0], hi[0] + 1) - t["origin"][0]) + off
                        n = np.clip(nd.astype(np.int64), 0, L - 2)
                        frac = nd - n
                        pol = (t["pol_h"] if h == 0 else t["pol_e"])[K]
                        f = np.array([self.prof[A][h][2][x] for x in range(lo[A], hi[A] + 1)]) if A == 0 else np.full(1, self.prof[A][h][2][lo[A]])
                        amp = _levi(I, A, K) * f / DX * normal * pol
                        if pol == 0.0:
                            continue
                        # the increment's factor: E gains (dt / eps0) of it, eta * H loses (eta dt / mu0)
                        amp = amp * (self.inp["dt"] / EPS0 if h == 0 else self.inp["dt"] * ETA / MU0)
                        at = tuple(slice(lo[d] - 1, hi[d]) if shape[d] > 1 else slice(0, 1) for d in (2, 1, 0))
                        self.planes[h].append((I, at, torch.tensor(n, device="cuda"), torch.tensor(frac, device="cuda"), torch.tensor(amp, device="cuda")))

    def _half(self, h, t):
        own, other = self.F[h], self.F[1 - h]
        sgn = 1 if h == 0 else -1
        dim = self.inp["dim"]
        source = self.inp["src"]
        if source and (source["target"] == "E") == (h == 0):
            at = source["pos"][::-1]
            own[source["comp"]][at] -= self.last
        new = {}
        for I in self.comps[h]:
            d = None
            for J in range(dim):
                K = 3 - I - J
                if I == J or K not in self.comps[1 - h]:
                    continue
                f = other[K]
                shift = list(self.inner)
                s = self.inner[2 - J]
                shift[2 - J] = slice(s.start - sgn, s.stop - sgn)
                raw = f[self.inner] - f[tuple(shift)]
                raw *= _levi(I, J, K) * sgn
                if d is None:
                    d = self.scale[h][J] * raw
                else:
                    d.addcmul_(self.scale[h][J].expand_as(raw), raw)
                for part in self.slabs[h][I, J]:
                    sl, B, C, G, psi = part
                    d[sl] += psi * G
                    part[4] = psi * B + C * raw[sl]
                del raw
            new[I] = d
        row = t if h == 0 else t + 1
        for I, at, n, frac, amp in self.planes[h]:
            tab = self.tabs[1 - h][row]  # the E half takes the 1D grid's H, the H half its E
            v = ((1.0 - frac) * tab[n] + frac * tab[n + 1]) * amp
            new[I][at] += v
        for I in self.comps[h]:
            e, d = own[I][self.inner], new.pop(I)
            if h == 1:
                e -= d
                continue
            for p in self.poles:
                d -= p["J"][I]
            d *= self.ie
            e += d
            for p in self.poles:
                j = p["J"][I]
                if p["P"][I] is not None:
                    p["P"][I] += j
                j *= p["a"]
                if isinstance(p["b"], torch.Tensor):
                    j.addcmul_(p["b"], e)
                else:
                    j.add_(e, alpha=p["b"])
                if p["P"][I] is not None:
                    j.add_(p["P"][I], alpha=-p["c"])
            del d
        if source and (source["target"] == "E") == (h == 0):
            v = float(source["vals"][t]) if t < len(source["vals"]) else 0.0
            self.last = v * (ETA if h == 1 else 1.0)
            own[source["comp"]][source["pos"][::-1]] += self.last
        for q, (comp, lo, hi) in enumerate(self.inp["dfts"]):
            if (comp < 3) != (h == 0):
                continue
            n = t + 1 if h == 0 else t + 1.5
            x = own[comp % 3][tuple(slice(l, u + 1) for l, u in zip(lo[::-1], hi[::-1]))]
            for f, freq in enumerate(self.inp["freqs"]):
                ang = -2.0 * math.pi * math.fmod(freq * n, 1.0)
                self.spectra[q][f] += x * complex(math.cos(ang), math.sin(ang)) / (ETA if h == 1 else 1.0)

    def run(self):
        for t in range(self.inp["steps"]):
            self._half(0, t)
            self._half(1, t)
        out = {"E" + "xyz"[c]: self.F[0][c] for c in self.comps[0]}
        for c in self.comps[1]:
            out["H" + "xyz"[c]] = self.F[1][c] if self.inp["f32"] else self.F[1][c] / ETA
        for q, x in enumerate(self.spectra):
            out["dft%d" % q] = x.reshape(len(self.inp["freqs"]), -1)
        return out


def _exact_adjoint(case, seed):
    """J and dJ/deps by torch's reverse mode over segments of the steps."""
    d, nx, ny, dt = _design(case, seed), case["nx"], case["ny"], _dt(TM)
    dev = dict(dtype=torch.float64, device="cuda")
    px, py = _grading(nx, case["npml"], dt, DX), _grading(ny, case["npml"], dt, DX)
    ce, ch = dt / (EPS0 * ETA * DX), ETA * dt / (MU0 * DX)
    co = []
    for h, c in ((0, ce), (1, ch)):
        x = [torch.tensor(v[1:-1], **dev)[None, :] for v in px[h]]
        y = [torch.tensor(v[1:-1], **dev)[:, None] for v in py[h]]
        co.append((x[0], c * x[1], c * x[2], x[3], y[0], c * y[1], c * y[2], y[3]))
    (x0, y0, _), (x1, y1, _) = d["design"]
    (pc, j0, _), (_, j1, _) = d["probe"]
    eps = torch.ones((ny - 2, nx - 2), **dev)
    eps[y0 - 1:y1, x0 - 1:x1] = torch.tensor(d["eps"][0, y0:y1 + 1, x0:x1 + 1], **dev)
    pad = torch.nn.functional.pad

    def step(s, ie, v_old, v):
        ez, hx, hy, a, b, c, e = s  # inner cells; a, b: E integrators along x, y; c, e: H's along y, x
        Bx, Cx, Fx, Gx, By, Cy, Fy, Gy = co[0]
        rx = hy - pad(hy, (1, 0))[:, :-1]
        ry = pad(hx, (0, 0, 1, 0))[:-1] - hx
        line = torch.zeros_like(ez)
        line[:, d["col"] - 1] = 1.0
        ez = ez - v_old * line + ie * (Fx * rx + Fy * ry + a * Gx + b * Gy) + v * line
        a, b = Bx * a + Cx * rx, By * b + Cy * ry
        Bx, Cx, Fx, Gx, By, Cy, Fy, Gy = co[1]
        ry = pad(ez, (0, 0, 0, 1))[1:] - ez
        rx = ez - pad(ez, (0, 1))[:, 1:]
        hx, hy = hx - (Fy * ry + c * Gy), hy - (Fx * rx + e * Gx)
        return ez, hx, hy, a, b, By * c + Cy * ry, Bx * e + Cx * rx

    def phase(t):
        ang = -2.0 * math.pi * math.fmod(d["freq"] * (t + 1), 1.0)
        return math.cos(ang), math.sin(ang)

    vals, N, seg = d["vals"], case["steps"], 50
    state = tuple(torch.zeros((ny - 2, nx - 2), **dev) for _ in range(7))
    saved, X = [], torch.zeros((2, j1 - j0 + 1), **dev)
    with torch.no_grad():
        for t in range(N):
            if t % seg == 0:
                saved.append(state)
            state = step(state, 1.0 / eps, vals[t - 1] if t else 0.0, vals[t])
            c, s = phase(t)
            p = state[0][j0 - 1:j1, pc - 1]
            X[0] += p * c
            X[1] += p * s
    J = float((X ** 2).sum())
    grad, lam = torch.zeros_like(eps), tuple(torch.zeros_like(eps) for _ in range(7))
    for k in range(len(saved) - 1, -1, -1):
        first = tuple(x.clone().requires_grad_() for x in saved[k])
        e = eps.clone().requires_grad_()
        s, part, ie = first, 0.0, 1.0 / e
        for t in range(k * seg, min(N, (k + 1) * seg)):
            s = step(s, ie, vals[t - 1] if t else 0.0, vals[t])
            c, sn = phase(t)
            part = part + (s[0][j0 - 1:j1, pc - 1] * (2.0 * (X[0] * c + X[1] * sn))).sum()
        total = part + sum((x * y).sum() for x, y in zip(s, lam))
        got = torch.autograd.grad(total, (*first, e))
        lam, grad = got[:7], grad + got[7]
    return {"J": J, "grad": grad[y0 - 1:y1, x0 - 1:x1].cpu().numpy()}


def exact(case, seed):
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed)
    if case["kind"] == "grid":
        return _Exact(_inputs(case, seed), seed).run()
    parts = [_Exact(_inputs(c, seed + 7919 * (q + 1)), seed + 7919 * (q + 1)).run() for q, c in enumerate(_config3(case, seed))]
    return {n: torch.cat([p[n].reshape(-1) for p in parts]) for n in parts[0]}
