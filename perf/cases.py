"""The work a user of the library has it do, as cases that can be timed and checked.

Every case goes through the package's public entry points (Context, Ensemble and
the gradients) with particles of its own making: cell by cell as the loader leaves
them, uniform inside each cell, drifting Maxwellians. `exact` restates the same
runs in plain torch, 64 bits, on the GPU.

Kinds:
  es        one electrostatic run from its loaded state: the particles are put
            back, aw_init, `steps` steps with every step's diagnostics to the host
  darwin    `steps` more steps of a Darwin run that is under way (its periodic
            re-sorts included as they fall due)
  yee       the same for a full-Maxwell Yee run
  ensemble  `steps` steps of several runs of uneven size advanced together
  grad_es, grad_darwin   one gradient of the final field energy
  operators one unfused Darwin step: every operator called by itself, as a host
            program that owns its own step does
  resort    one spatial re-sort of particles that have mixed
"""
import math

import numpy as np
import torch

import arcwarden_b200 as aw

PKEYS = ("x", "y", "ux", "uy", "uz", "w")
TOTAL = 33_554_432          # particles of the largest listed run
_stream = None


def stream():
    """The one stream of the program (a user's run loop has one)."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


# ---- the cases -----------------------------------------------------------------
def listed():
    return [
        # the smallest runs of a parameter scan: 65 k particles, where launches and latency count
        dict(name="es 64x64", kind="es", nx=64, ny=64, dx=1.0, ppc=16, vth=0.03, vd=0.2, bz=0.0, dt=0.1, steps=50),
        # the electrostatic two-stream benchmark (4.2 M particles)
        dict(name="es 256x256", kind="es", nx=256, ny=256, dx=1.0, ppc=64, vth=0.01, vd=0.2, bz=0.0, dt=0.1, steps=20),
        # an electrostatic run off the powers of two: odd grid, cell size 0.3, magnetised, ragged count
        dict(name="es 375x225 magnetised", kind="es", nx=375, ny=225, dx=0.3, ppc=50, vth=0.05, vd=0.1, bz=0.5, dt=0.1,
             steps=20),
        # the Darwin Weibel benchmark (16.8 M particles, 64 per cell)
        dict(name="darwin weibel 512x512", kind="darwin", nx=512, ny=512, dx=0.5, ppc=64, vth=0.05, vz=0.2, b0=0.0,
             pump=False, dt=0.05, c=1.0, steps=10),
        # the magnetised Darwin whistler benchmark, the largest single run (33.6 M particles, 256 per cell)
        dict(name="darwin whistler 1024x128", kind="darwin", nx=1024, ny=128, dx=0.25, ppc=256, vth=0.019, vz=0.019,
             b0=0.5, pump=True, dt=0.05, c=1.0, steps=10),
        # the whistler decks' shape: a grid one cell high, many particles per cell
        dict(name="darwin 512x1", kind="darwin", nx=512, ny=1, dx=2.0, ppc=512, vth=0.5, vz=0.5, b0=0.3, pump=True,
             dt=0.02, c=25.0, steps=20),
        # a Darwin run off the powers of two, few particles per cell
        dict(name="darwin 300x180", kind="darwin", nx=300, ny=180, dx=0.3, ppc=25, vth=0.05, vz=0.1, b0=0.3, pump=False,
             dt=0.05, c=1.0, steps=10),
        # the Yee whistler-anisotropy benchmark at 100 of its 400 particles per cell, current filter on
        dict(name="yee 625x625", kind="yee", nx=625, ny=625, dx=0.0216, ppc=100, vth=0.03752, vx=0.01678, b0=0.25,
             dt=0.0145, jfilter=3, steps=5),
        # a batched parameter scan: 12 runs of uneven size, both models
        dict(name="ensemble of 12", kind="ensemble", nruns=12, scan=0, steps=10),
        # one gradient of an electrostatic run (optimising initial conditions)
        dict(name="gradient es 256x256", kind="grad_es", nx=256, ny=256, dx=1.0, ppc=16, vth=0.01, vd=0.2, bz=0.0,
             dt=0.1, steps=40, every=10),
        # one gradient of a Darwin run with its pump amplitude
        dict(name="gradient darwin 256x256", kind="grad_darwin", nx=256, ny=256, dx=0.5, ppc=16, vth=0.05, vz=0.2,
             b0=0.3, pump=True, dt=0.05, c=1.0, steps=20, every=10),
        # the operators one by one, at the size of the reference's kernel benchmark
        dict(name="operators 256x256", kind="operators", nx=256, ny=256, dx=0.5, ppc=64, vth=0.05, vz=0.2, b0=0.3,
             pump=False, dt=0.05, c=1.0, steps=1),
    ]


SIDES = (32, 40, 48, 50, 60, 63, 64, 75, 80, 96, 105, 108, 120, 125, 128, 135, 150, 160, 175, 180, 192, 200, 225, 240, 256,
         270, 288, 300, 315, 320, 360, 375, 384, 400, 432, 450, 480, 512, 576, 600, 625, 640, 720, 768, 900, 1024)


def _grid(rng, most, lo=32):
    """A grid of FFT-friendly sides with about a log-uniform number of cells, at most `most`."""
    cells = math.exp(rng.uniform(math.log(lo * lo), math.log(most)))
    skew = math.exp(rng.uniform(-0.7, 1.2))
    near = lambda v: min(SIDES, key=lambda s: abs(math.log(s / v)))  # noqa: E731
    nx, ny = near(math.sqrt(cells) * math.sqrt(skew)), near(math.sqrt(cells) / math.sqrt(skew))
    while nx * ny > most:
        nx, ny = SIDES[max(0, SIDES.index(nx) - 1)], SIDES[max(0, SIDES.index(ny) - 1)]
    return nx, ny


def _ppc(rng, cells, most, lo=8, hi=400):
    return max(lo, min(hi, int(most // cells), int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("es", "es", "darwin", "darwin", "darwin", "yee", "ensemble", "grad_es", "grad_darwin", "operators",
                       "resort"))
    vth = round(math.exp(rng.uniform(math.log(0.01), math.log(0.1))), 4)
    dx = rng.choice((0.25, 0.3, 0.5, 1.0))
    if kind == "es":
        nx, ny = _grid(rng, 512 * 512)
        ppc = _ppc(rng, nx * ny, TOTAL // 2) & ~1
        return dict(kind=kind, nx=nx, ny=ny, dx=dx, ppc=ppc, vth=vth, vd=round(rng.uniform(0.0, 0.3), 3),
                    bz=rng.choice((0.0, round(rng.uniform(0.2, 1.0), 3))), dt=0.1, steps=rng.choice((10, 15, 20)))
    if kind in ("darwin", "operators", "resort"):
        nx, ny = _grid(rng, 512 * 512)
        if kind == "darwin" and rng.random() < 0.15:
            nx, ny = rng.choice((200, 256, 512, 1000)), 1
        ppc = _ppc(rng, nx * ny, TOTAL // 2 if kind == "darwin" else TOTAL // 4, hi=600 if ny == 1 else 400)
        return dict(kind=kind, nx=nx, ny=ny, dx=dx, ppc=ppc, vth=vth, vz=round(vth * rng.uniform(1.0, 4.0), 4),
                    b0=rng.choice((0.0, round(rng.uniform(0.1, 0.6), 3))), pump=rng.random() < 0.4, dt=0.05, c=1.0,
                    steps=1 if kind != "darwin" else rng.choice((5, 8, 10)))
    if kind == "yee":
        nx, ny = _grid(rng, 512 * 512)
        dx = rng.choice((0.02, 0.025, 0.03125))
        return dict(kind=kind, nx=nx, ny=ny, dx=dx, ppc=_ppc(rng, nx * ny, TOTAL // 2), vth=vth, vx=round(vth / 2, 4),
                    b0=round(rng.uniform(0.0, 0.5), 3), dt=0.65 * dx, jfilter=rng.choice((0, 1, 3)), steps=rng.choice((2, 4)))
    if kind == "ensemble":
        return dict(kind=kind, nruns=rng.choice((3, 5, 8, 12)), scan=rng.randrange(1, 1000), steps=rng.choice((5, 10)))
    nx, ny = _grid(rng, 256 * 256)
    every = rng.choice((4, 5, 7, 10))
    case = dict(kind=kind, nx=nx, ny=ny, dx=dx, ppc=_ppc(rng, nx * ny, 1 << 20, hi=64) & ~1, vth=vth)
    if kind == "grad_es":
        return dict(case, vd=round(rng.uniform(0.0, 0.3), 3), bz=rng.choice((0.0, 0.4)), dt=0.1, every=every,
                    steps=rng.choice((20, 25, 40)))
    return dict(case, vz=round(2 * vth, 4), b0=0.3, pump=True, dt=0.05, c=1.0, every=every, steps=rng.choice((10, 15, 20)))


# ---- inputs ----------------------------------------------------------------------
def count(case):
    return case["nx"] * case["ny"] * case["ppc"]


def _load(case, seed, beams):
    """Particles in cell order, `beams` species one after the other, as the loader leaves them."""
    nx, ny, ppc, dx = case["nx"], case["ny"], case["ppc"], case["dx"]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    f32 = dict(dtype=torch.float32, device="cuda")
    n = nx * ny * ppc
    P = {k: torch.empty(n, **f32) for k in PKEYS}
    per = ppc // len(beams)
    at = 0
    for s, (uth, ufl) in enumerate(beams):
        m = per if s + 1 < len(beams) else ppc - at // (nx * ny)
        cell = torch.arange(nx * ny, device="cuda").repeat_interleave(m)
        sl = slice(at, at + m * nx * ny)
        for k, base, top in (("x", cell % nx, nx), ("y", cell // nx, ny)):
            v = base.to(torch.float32) + torch.rand(base.shape, generator=g, **f32)
            P[k][sl] = v.clamp_(max=float(np.nextafter(np.float32(top), np.float32(0))))
        for d, k in enumerate(("ux", "uy", "uz")):
            P[k][sl] = torch.randn(cell.shape, generator=g, **f32).mul_(uth[d]).add_(ufl[d])
        at += m * nx * ny
    P["w"].fill_(dx * dx / ppc)
    return P


def _beams(case):
    if "vd" in case:
        return [((case["vth"],) * 3, (case["vd"], 0.0, 0.0)), ((case["vth"],) * 3, (-case["vd"], 0.0, 0.0))]
    vx = case.get("vx", case["vth"])
    return [((vx, case["vth"], case.get("vz", case["vth"])), (0.0, 0.0, 0.0))]


def _b0(case):
    if case["kind"] in ("es", "grad_es"):
        return (0.0, 0.0, case["bz"])
    if case["kind"] == "yee":
        return (case["b0"], 0.0, 0.0)
    th = math.radians(30.0)
    return (case["b0"] * math.cos(th), case["b0"] * math.sin(th), 0.0)


def _pump(case):
    if not case.get("pump"):
        return None
    return dict(ex=1e-3, ey=2e-3, ez=-2e-3, k0=2 * math.pi * 4 / (case["nx"] * case["dx"]), w0=0.05, trmp=1.0, toff=1.0e9)


def _model(case):
    return {"es": aw.AW_MODEL_ES, "grad_es": aw.AW_MODEL_ES, "yee": aw.AW_MODEL_YEE}.get(case["kind"], aw.AW_MODEL_DARWIN)


class Run:
    """A context with the particle, source and field arrays its program owns."""

    def __init__(self, case, seed):
        nx, ny, dx = case["nx"], case["ny"], case["dx"]
        self.case, self.n, self.step = case, count(case), 0
        self.P = _load(case, seed, _beams(case))
        self.cell = torch.empty(self.n, dtype=torch.int32, device="cuda")
        self.ctx = aw.Context(nx, ny, nx * dx, ny * dx, dt=case["dt"], c=case.get("c", 1.0), B0=_b0(case),
                              model=_model(case), stream=stream().cuda_stream, pump=_pump(case))
        self.ctx.bind_particles(*(self.P[k] for k in PKEYS), self.cell)
        self.G = {k: torch.zeros(ny, nx, dtype=torch.float32, device="cuda") for k in aw.SOURCE_NAMES + aw.FIELD_NAMES}
        self.ctx.bind_sources(**{k: self.G[k] for k in aw.SOURCE_NAMES})
        self.ctx.bind_fields(**{k: self.G[k] for k in aw.FIELD_NAMES})
        torch.cuda.synchronize()

    def outputs(self, grids, keys=PKEYS[:5]):
        return {**{k: self.P[k] for k in keys}, **{k: self.G[k] for k in grids}}

    def __del__(self):
        if getattr(self, "ctx", None) is not None:
            torch.cuda.synchronize()
            self.ctx.close()


class _Device:
    """A device array of the library's, for torch."""

    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f4", "data": (ptr, False), "version": 3}


class Scan:
    """An ensemble whose runs start from this program's own particles."""

    def __init__(self, case, seed):
        self.runs, self.steps = _scan(case), case["steps"]
        specs = []
        for r in self.runs:
            sp = [dict(ppc=r["ppc"] // 2, density=0.5, uth=(r["vth"],) * 3, ufl=(r["vd"] * s, 0.0, 0.0)) for s in (1, -1)]
            specs.append(aw.run_spec(_model(r), r["nx"], r["ny"], r["nx"] * r["dx"], r["ny"] * r["dx"], sp, seed=0,
                                     dt=r["dt"], B0=_b0(r)))
        self.ens = aw.Ensemble(specs, stream=stream().cuda_stream)
        self.parts = []
        for k, r in enumerate(self.runs):
            ptr, n = self.ens.particles(k)
            mine, theirs = _load(r, seed + 1000 * k, _beams(r)), {}
            for key in PKEYS:
                theirs[key] = torch.as_tensor(_Device(ptr[key], n), device="cuda")
                theirs[key].copy_(mine[key])
            self.parts.append(theirs)
        torch.cuda.synchronize()
        self.ens.init()

    def __del__(self):
        if getattr(self, "ens", None) is not None:
            torch.cuda.synchronize()
            self.ens.close()


def _scan(case):
    rng = np.random.default_rng(case["scan"])
    runs = []
    for r in range(case["nruns"]):
        side, ppc = int(rng.choice((64, 128, 256))), int(rng.choice((16, 64, 256), p=(0.4, 0.4, 0.2)))
        kind = "es" if r % 2 == 0 else "darwin"
        b = float(rng.uniform(0.2, 1.0)) if (r // 2) % 2 else 0.0
        runs.append(dict(kind=kind, nx=side, ny=side, dx=1.0, ppc=ppc, vth=float(math.exp(rng.uniform(math.log(0.01), math.log(0.1)))),
                         vd=float(rng.uniform(0.0, 0.3)), bz=b, b0=b, dt=0.1 if kind == "es" else 0.05, c=1.0))
    return runs


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        return Scan(case, seed)
    r = Run(case, seed)
    if kind in ("es", "resort"):
        r.start = {k: r.P[k].clone() for k in PKEYS[:5]}
        r.diag = torch.zeros(case["steps"], 8, dtype=torch.float64).pin_memory()
    if kind == "resort":           # a run's particles, 200 steps of free motion after the load
        for k, u in (("x", "ux"), ("y", "uy")):
            m = float(case["nx"] if k == "x" else case["ny"])
            v = torch.remainder(r.P[k] + r.P[u] * (200 * case["dt"] / case["dx"]), m)
            r.start[k] = torch.where(v < m, v, torch.zeros_like(v))
    if kind == "yee":
        r.ctx.set_current_filter(case["jfilter"])
    if kind in ("darwin", "yee"):
        r.ctx.init()
    if kind in ("grad_es", "grad_darwin"):
        r.du = [torch.zeros(r.n, dtype=torch.float32, device="cuda") for _ in range(3)]
    if kind == "operators":
        X = torch.arange(case["nx"], device="cuda") * (2 * math.pi / case["nx"])
        Y = torch.arange(case["ny"], device="cuda")[:, None] * (2 * math.pi / case["ny"])
        b = _b0(case)
        r.in_fields = {"Ex": 0.01 * torch.sin(X + 0 * Y), "Ey": 0.01 * torch.cos(Y + 0 * X), "Ez": 0.005 * torch.sin(X + Y),
                       "Bx": b[0] + 0.01 * torch.cos(X + 0 * Y), "By": b[1] + 0.02 * torch.sin(Y + 0 * X), "Bz": 0.1 + 0 * (X + Y)}
        r.start = {k: r.P[k].clone() for k in PKEYS[:5]}
    torch.cuda.synchronize()
    return r


# ---- one pass ----------------------------------------------------------------------
GRIDS_ES = ("rho", "Ex", "Ey")
GRIDS_EM = ("Ex", "Ey", "Ez", "Bx", "By", "Bz")
SOURCES = ("rho", "Jx", "Jy", "Jz", "amu0", "amu1", "amu2", "amu3")
DCU = ("dcux", "dcuy", "dcuz")


def run(state):
    if isinstance(state, Scan):
        state.ens.run(state.steps)
        # copies: the particle arrays are the ensemble's own and go with it
        with torch.cuda.stream(stream()):
            return [{k: p[k].clone() for k in PKEYS[:5]} for p in state.parts]
    return {"es": _run_es, "darwin": _run_on, "yee": _run_on, "grad_es": _run_grad, "grad_darwin": _run_grad,
            "operators": _run_operators, "resort": _run_resort}[state.case["kind"]](state)


def _restore(r):
    with torch.cuda.stream(stream()):
        for k, v in r.start.items():
            r.P[k].copy_(v)


def _run_es(r):
    _restore(r)
    r.ctx.init()
    r.ctx.run_diag(0, r.case["steps"], r.diag.data_ptr())
    stream().synchronize()
    return {**r.outputs(GRIDS_ES), "diag": r.diag[:, :7].clone()}


def _run_on(r):
    r.ctx.run(r.step, r.case["steps"])
    r.step += r.case["steps"]
    return r.outputs(GRIDS_EM)


def _run_grad(r):
    if r.case["kind"] == "grad_es":
        loss, dp = r.ctx.grad_es(r.case["steps"], r.case["every"], *r.du), 0.0
    else:
        loss, dp = r.ctx.grad_darwin(r.case["steps"], r.case["every"], *r.du)
    return {"loss": loss, "dpump": dp, "du": list(r.du)}


def _run_operators(r):
    c, G = r.ctx, r.G
    _restore(r)
    with torch.cuda.stream(stream()):
        for k, v in r.in_fields.items():
            G[k].copy_(v)
        for k in SOURCES + DCU:
            G[k].zero_()
    c.deposit_rho_j()
    c.deposit_amu()
    c.solve_darwin_el_b()
    c.add_b0()
    with torch.cuda.stream(stream()):
        G["Ex"].copy_(G["ELx"])
        G["Ey"].copy_(G["ELy"])
        G["Ez"].zero_()
    c.deposit_dcu()
    c.solve_darwin_et()
    c.form_e(1.0)
    c.push_em()
    c.migrate()
    return r.outputs(SOURCES + DCU + GRIDS_EM)


def _run_resort(r):
    _restore(r)
    r.ctx.resort()
    return r.outputs((), PKEYS)


# ---- what a pass cannot do without -------------------------------------------------------
def work(case):
    """Bytes: the particle state in and out of every step (x y ux uy uz w read, x y
    ux uy uz written; the Darwin dcu deposit reads it once more, because the push
    needs the field that deposit makes) and the grids. A gradient runs each step
    forward and transposed: the transposed step reads the state and reads and
    writes the five cotangents, for Darwin once for each of its three fields'
    solves. FLOPs: the gathers, pushes and deposits."""
    kind = case["kind"]
    if kind == "ensemble":
        parts = [work(dict(r, steps=case["steps"])) for r in _scan(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n, nc, s = count(case), case["nx"] * case["ny"], case["steps"]
    if kind == "es":
        return {"bytes": s * (44 * n + 12 * nc), "flops": s * 110 * n}
    if kind == "darwin":
        return {"bytes": s * (68 * n + 56 * nc), "flops": s * 330 * n}
    if kind == "yee":
        return {"bytes": s * (44 * n + 48 * nc), "flops": s * 350 * n}
    if kind == "grad_es":
        return {"bytes": s * (44 + 24 + 40) * n, "flops": s * 330 * n}
    if kind == "grad_darwin":
        return {"bytes": s * (68 + 3 * 64) * n, "flops": s * 1200 * n}
    if kind == "operators":
        return {"bytes": (24 + 24 + 24 + 44) * n + 150 * nc, "flops": 330 * n}
    return {"bytes": 2 * 28 * n, "flops": 0}


def tolerance(case):
    """About four times what a run in 64 bits differs by (measured, see exact).
    Particles and fields are 32-bit; a position in the hundreds carries a rounding
    of 3e-5 cells per step, which the noise part of E (a few per cent of the charge
    density's gradient) shows at 1e-4, the Yee current (differences of shapes) at
    7e-4, and a gradient, which carries it through every step, at 1e-2."""
    return {"resort": "exact", "operators": {"rel": 1e-4, "max": 1e-2}, "yee": {"rel": 3e-3, "max": 0.1},
            "grad_es": {"rel": 0.03, "max": 0.9}, "grad_darwin": {"rel": 0.02, "max": 0.9}}.get(
                case["kind"], {"rel": 5e-4, "max": 5e-2})


# ---- the same in 64 bits ----------------------------------------------------------------
class Grid64:
    """CIC, the spectral solves and the pushes in float64 torch; differentiable."""

    def __init__(self, case):
        self.nx, self.ny, self.dx, self.dt = case["nx"], case["ny"], case["dx"], case["dt"]
        self.area, self.qm, self.c, self.b0 = self.dx * self.dx, -1.0, case.get("c", 1.0), _b0(case)
        self.pump = _pump(case)
        d = dict(dtype=torch.float64, device="cuda")
        kx = torch.arange(self.nx // 2 + 1, **d) * (2 * math.pi / (self.nx * self.dx))
        m = torch.arange(self.ny, **d)
        ky = (torch.where(m <= self.ny // 2, m, m - self.ny) * (2 * math.pi / (self.ny * self.dx)))[:, None]
        k2 = kx * kx + ky * ky
        keep = (k2 > 0).to(torch.float64)
        if self.nx % 2 == 0:
            keep[:, self.nx // 2] = 0
        if self.ny % 2 == 0:
            keep[self.ny // 2, :] = 0
        self.kx, self.ky, self.k2 = kx, ky, torch.where(k2 > 0, k2, torch.ones_like(k2))
        self.ge = keep / self.k2
        self.gb = self.ge / self.c ** 2
        self.gt = keep / (self.c ** 2 * self.k2 + 1.0)

    def stencil(self, x, y):
        i, j = torch.floor(x.detach()), torch.floor(y.detach())
        fx, fy = x - i, y - j
        i, j = i.to(torch.int64) % self.nx, j.to(torch.int64) % self.ny
        i1, j1 = (i + 1) % self.nx, (j + 1) % self.ny
        return ((j * self.nx + i, (1 - fx) * (1 - fy)), (j * self.nx + i1, fx * (1 - fy)),
                (j1 * self.nx + i, (1 - fx) * fy), (j1 * self.nx + i1, fx * fy))

    def deposit(self, st, v):
        a = torch.zeros(self.nx * self.ny, dtype=torch.float64, device="cuda")
        for c, w in st:
            a = a.index_add(0, c, w * v)
        return a.view(self.ny, self.nx)

    def gather(self, st, f):
        f = f.reshape(-1)
        return sum(w * f[c] for c, w in st)

    def real(self, f):
        return torch.fft.irfft2(f, s=(self.ny, self.nx))

    def solve_e(self, rho):
        r = torch.fft.rfft2(rho) * self.ge
        return self.real(-1j * self.kx * r), self.real(-1j * self.ky * r)

    def solve_b(self, J):
        j = [torch.fft.rfft2(a) * self.gb for a in J]
        return (self.real(1j * self.ky * j[2]), self.real(-1j * self.kx * j[2]),
                self.real(1j * (self.kx * j[1] - self.ky * j[0])))

    def solve_et(self, dcu, amu):
        d, a = [torch.fft.rfft2(v) for v in dcu], [torch.fft.rfft2(v) for v in amu]
        S = (self.kx * a[0] + self.ky * a[1], self.kx * a[1] - self.ky * a[0], self.kx * a[2] + self.ky * a[3])
        J = [d[k] - 1j * S[k] for k in range(3)]
        kd = (self.kx * J[0] + self.ky * J[1]) / self.k2
        return [self.real(-self.gt * v) for v in (J[0] - self.kx * kd, J[1] - self.ky * kd, J[2])]

    def pump_at(self, t):
        p = self.pump
        if not p:
            return (0.0, 0.0, 0.0)
        r = min(1.0, t / p["trmp"])
        th = p["k0"] * torch.arange(self.nx, dtype=torch.float64, device="cuda") * self.dx - p["w0"] * t
        return (p["ex"] * torch.cos(th) * r, -p["ey"] * torch.sin(th) * r, p["ez"] * torch.cos(th) * r)

    @staticmethod
    def cross(a, b):
        return (a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0])

    def boris(self, u, e, b, dt):
        h = self.qm * 0.5 * dt
        u = [u[d] + h * e[d] for d in range(3)]
        t = [h * b[d] for d in range(3)]
        t2 = t[0] * t[0] + t[1] * t[1] + t[2] * t[2]
        s = [2 * v / (1 + t2) for v in t]
        up = [a + b_ for a, b_ in zip(u, self.cross(u, t))]
        u = [a + b_ for a, b_ in zip(u, self.cross(up, s))]
        return [u[d] + h * e[d] for d in range(3)]

    def move(self, x, y, u):
        x, y = x + u[0] * (self.dt / self.dx), y + u[1] * (self.dt / self.dx)
        return x - torch.floor(x.detach() / self.nx) * self.nx, y - torch.floor(y.detach() / self.ny) * self.ny

    def es_fields(self, x, y, w):
        st = self.stencil(x, y)
        rho = self.deposit(st, self.qm / self.area * w)
        return st, rho, self.solve_e(rho)

    def es_push(self, st, E, u, dt):
        e = (self.gather(st, E[0]), self.gather(st, E[1]), torch.zeros_like(u[0]))
        return self.boris(u, e, self.b0, dt)

    def sources(self, st, u, w):
        q = self.qm / self.area * w
        amu = (0.5 * (u[0] * u[0] - u[1] * u[1]), u[0] * u[1], u[2] * u[0], u[2] * u[1])
        return self.deposit(st, q), [self.deposit(st, q * v) for v in u], [self.deposit(st, q * v) for v in amu]

    def dcu(self, st, F, B, u, w):
        q = self.qm * self.qm / self.area * w
        b = [self.gather(st, v) for v in B]
        c = self.cross(u, b)
        return [self.deposit(st, q * (self.gather(st, F[d]) + c[d])) for d in range(3)]

    def darwin_fields(self, x, y, u, w, t, amp=1.0):
        st = self.stencil(x, y)
        rho, J, amu = self.sources(st, u, w)
        el, b = self.solve_e(rho), self.solve_b(J)
        B = [b[d] + self.b0[d] for d in range(3)]
        p = [amp * v for v in self.pump_at(t)]
        zero = torch.zeros_like(rho)
        F = [el[0] + p[0], el[1] + p[1], zero + p[2]]
        et = self.solve_et(self.dcu(st, F, B, u, w), amu)
        return st, [el[0] + et[0] + p[0], el[1] + et[1] + p[1], et[2] + p[2]], B


def _state64(P):
    return P["x"].double(), P["y"].double(), [P[k].double() for k in ("ux", "uy", "uz")], P["w"].double()


def _exact_es(case, P):
    g = Grid64(case)
    x, y, u, w = _state64(P)
    st, rho, E = g.es_fields(x, y, w)
    u = g.es_push(st, E, u, -0.5 * g.dt)
    diag = []
    for _ in range(case["steps"]):
        st, rho, E = g.es_fields(x, y, w)
        u = g.es_push(st, E, u, g.dt)
        x, y = g.move(x, y, u)
        e2 = E[0] ** 2 + E[1] ** 2
        diag.append([0.5 * (w * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2)).sum(), 0.5 * e2.sum() * g.area, rho.sum() * g.area,
                     e2.max().sqrt()] + [(w * v).sum() for v in u])
    return {"x": x, "y": y, "ux": u[0], "uy": u[1], "uz": u[2], "rho": rho, "Ex": E[0], "Ey": E[1],
            "diag": torch.tensor([[float(v) for v in d] for d in diag], dtype=torch.float64)}


def _exact_darwin(case, P):
    g = Grid64(case)
    x, y, u, w = _state64(P)
    for s in range(case["steps"]):
        st, E, B = g.darwin_fields(x, y, u, w, s * g.dt)
        u = g.boris(u, [g.gather(st, v) for v in E], [g.gather(st, v) for v in B], g.dt)
        x, y = g.move(x, y, u)
        del st
    return dict(zip(PKEYS[:5] + GRIDS_EM, [x, y, *u, *E, *B]))


def _exact_operators(case, P):
    g = Grid64(case)
    x, y, u, w = _state64(P)
    st = g.stencil(x, y)
    rho, J, amu = g.sources(st, u, w)
    el, b = g.solve_e(rho), g.solve_b(J)
    B = [b[d] + g.b0[d] for d in range(3)]
    dcu = g.dcu(st, [el[0], el[1], torch.zeros_like(rho)], B, u, w)
    et = g.solve_et(dcu, amu)
    E = [el[0] + et[0], el[1] + et[1], et[2]]
    u = g.boris(u, [g.gather(st, v) for v in E], [g.gather(st, v) for v in B], g.dt)
    x, y = g.move(x, y, u)
    return dict(zip(PKEYS[:5] + SOURCES + DCU + GRIDS_EM, [x, y, *u, rho, *J, *amu, *dcu, *E, *B]))


def _exact_grad(case, P):
    g = Grid64(case)
    x, y, u, w = _state64(P)
    u0 = [v.requires_grad_() for v in u]
    amp = torch.ones((), dtype=torch.float64, device="cuda", requires_grad=True)
    es = case["kind"] == "grad_es"
    u = u0
    if es:
        st, _, E = g.es_fields(x, y, w)
        # the rollback is a transposed step of its own: its field is that of the initial positions, which do not depend on u
        u = g.es_push(st, [v.detach() for v in E], u, -0.5 * g.dt)
    for s in range(case["steps"]):
        if es:
            st, _, E = g.es_fields(x, y, w)
            u = g.es_push(st, E, u, g.dt)
        else:
            st, E, B = g.darwin_fields(x, y, u, w, s * g.dt, amp)
            u = g.boris(u, [g.gather(st, v) for v in E], [g.gather(st, v) for v in B], g.dt)
        x, y = g.move(x, y, u)
    loss = 0.5 * g.area * (E[0] ** 2 + E[1] ** 2).sum()
    got = torch.autograd.grad(loss, u0 + [amp], allow_unused=True)
    return {"loss": float(loss.detach()), "dpump": 0.0 if es else float(got[3]), "du": [v.contiguous() for v in got[:3]]}


def _exact_yee(case, P):
    nx, ny, dx, dt = case["nx"], case["ny"], case["dx"], case["dt"]
    d = dict(dtype=torch.float64, device="cuda")
    f = {k: torch.zeros(ny, nx, **d) for k in GRIDS_EM}
    x, y, u, w = _state64(P)
    b0, qm, h = _b0(case), -1.0, -0.5 * dt
    off = {"Ex": (0.5, 0.0), "Ey": (0.0, 0.5), "Ez": (0.0, 0.0), "Bx": (0.0, 0.5), "By": (0.5, 0.0), "Bz": (0.5, 0.5)}
    right, up = (lambda a: torch.roll(a, -1, 1)), (lambda a: torch.roll(a, -1, 0))
    left, down = (lambda a: torch.roll(a, 1, 1)), (lambda a: torch.roll(a, 1, 0))

    def faraday(s):
        ez, ex, ey = f["Ez"], f["Ex"], f["Ey"]
        f["Bx"] = f["Bx"] - s * (up(ez) - ez) / dx
        f["By"] = f["By"] + s * (right(ez) - ez) / dx
        f["Bz"] = f["Bz"] - s * ((right(ey) - ey) / dx - (up(ex) - ex) / dx)

    def gather(k, x, y):
        xs, ys = x - off[k][0], y - off[k][1]
        i, j = torch.floor(xs), torch.floor(ys)
        fx, fy = xs - i, ys - j
        i, j = i.to(torch.int64) % nx, j.to(torch.int64) % ny
        i1, j1, a = (i + 1) % nx, (j + 1) % ny, f[k].reshape(-1)
        return ((1 - fx) * (1 - fy) * a[j * nx + i] + fx * (1 - fy) * a[j * nx + i1] + (1 - fx) * fy * a[j1 * nx + i]
                + fx * fy * a[j1 * nx + i1])

    def shapes(v, b):
        return [torch.clamp(1 - torch.abs(v - (b + k)), min=0) for k in range(3)]

    g = Grid64(case)
    block = 1 << 23                       # particles at a time
    for _ in range(case["steps"]):
        faraday(0.5 * dt)
        J = [torch.zeros(nx * ny, **d) for _ in range(3)]
        for lo in range(0, len(x), block):
            sl = slice(lo, lo + block)
            x0, y0 = x[sl], y[sl]
            e = [gather(k, x0, y0) for k in ("Ex", "Ey", "Ez")]
            b = [gather(k, x0, y0) + b0[m] for m, k in enumerate(("Bx", "By", "Bz"))]
            v = g.boris([a[sl] for a in u], e, b, dt)
            x1, y1 = x0 + v[0] * dt / dx, y0 + v[1] * dt / dx
            ib, jb = torch.floor(torch.minimum(x0, x1)), torch.floor(torch.minimum(y0, y1))
            sx, sy = shapes(x0, ib), shapes(y0, jb)
            tx, ty = [b_ - a for a, b_ in zip(sx, shapes(x1, ib))], [b_ - a for a, b_ in zip(sy, shapes(y1, jb))]
            q = qm * w[sl]
            ib, jb = ib.to(torch.int64), jb.to(torch.int64)
            for m in range(3):
                px = py = 0.0
                for k in range(3):
                    px = px + tx[k] * (sy[m] + 0.5 * ty[m])
                    py = py + ty[k] * (sx[m] + 0.5 * tx[m])
                    J[0].index_add_(0, (jb + m) % ny * nx + (ib + k) % nx, -q / (dt * dx) * px)
                    J[1].index_add_(0, (jb + k) % ny * nx + (ib + m) % nx, -q / (dt * dx) * py)
                    wz = sx[k] * sy[m] + 0.5 * (tx[k] * sy[m] + sx[k] * ty[m]) + tx[k] * ty[m] / 3
                    J[2].index_add_(0, (jb + m) % ny * nx + (ib + k) % nx, q * v[2] / (dx * dx) * wz)
            x[sl], y[sl] = x1 - torch.floor(x1 / nx) * nx, y1 - torch.floor(y1 / ny) * ny
            for a, b_ in zip(u, v):
                a[sl] = b_
        J = [a.view(ny, nx) for a in J]
        for _ in range(case["jfilter"]):
            J = [0.25 * left(a) + 0.5 * a + 0.25 * right(a) for a in J]
            J = [0.25 * down(a) + 0.5 * a + 0.25 * up(a) for a in J]
        faraday(0.5 * dt)
        f["Ex"] = f["Ex"] + dt * ((f["Bz"] - down(f["Bz"])) / dx - J[0])
        f["Ey"] = f["Ey"] + dt * (-(f["Bz"] - left(f["Bz"])) / dx - J[1])
        f["Ez"] = f["Ez"] + dt * ((f["By"] - left(f["By"])) / dx - (f["Bx"] - down(f["Bx"])) / dx - J[2])
    return dict(zip(PKEYS[:5], [x, y, *u]), **f)


def exact(case, seed):
    kind = case["kind"]
    if kind == "resort":
        return None                       # a permutation: nothing is computed
    if kind == "ensemble":
        out = []
        for k, r in enumerate(_scan(case)):
            r = dict(r, steps=case["steps"])
            got = (_exact_es if r["kind"] == "es" else _exact_darwin)(r, _load(r, seed + 1000 * k, _beams(r)))
            out.append({key: got[key] for key in PKEYS[:5]})
        return out
    P = _load(case, seed, _beams(case))
    return {"es": _exact_es, "darwin": _exact_darwin, "yee": _exact_yee, "grad_es": _exact_grad, "grad_darwin": _exact_grad,
            "operators": _exact_operators}[kind](case, P)
