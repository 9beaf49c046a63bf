"""The three-kernel grid solves against FP64 (numpy), over the radices and shapes they
take: powers of two, odd sides, every small factor, non-square, the longest rows and
columns, and a side the passes do not take (the library transforms)."""
import numpy as np
import pytest

from gpu_helpers import Setup

pytestmark = pytest.mark.gpu

# 1e-5 of the largest value is the solves' bar (the reference's metric); the FP32
# transforms are at a few 1e-7 sqrt(log N) of it.
SHAPES = [(64, 64), (48, 50), (75, 63), (105, 49), (70, 54), (128, 1024), (1024, 64), (375, 225), (98, 343), (62, 66)]


def solve64(nx, ny, L, rho, J):
    kx = 2 * np.pi / L[0] * np.arange(nx // 2 + 1)
    m = np.arange(ny)
    ky = (2 * np.pi / L[1] * np.where(m <= ny // 2, m, m - ny))[:, None]
    k2 = kx * kx + ky * ky
    keep = (k2 > 0).astype(float)
    if nx % 2 == 0:
        keep[:, nx // 2] = 0
    if ny % 2 == 0:
        keep[ny // 2, :] = 0
    g = keep / np.where(k2 > 0, k2, 1.0)
    r = np.fft.rfft2(rho)
    j = [np.fft.rfft2(a) for a in J]
    inv = lambda a: np.fft.irfft2(a, s=(ny, nx))  # noqa: E731
    return (inv(-1j * kx * g * r), inv(-1j * ky * g * r), inv(1j * g * ky * j[2]), inv(-1j * g * kx * j[2]),
            inv(1j * g * (kx * j[1] - ky * j[0])))


@pytest.mark.parametrize("nx,ny", SHAPES)
def test_solves_match_fp64(torch_cuda, aw, nx, ny):
    Lx, Ly = 0.3 * nx, 0.2 * ny
    s = Setup(torch_cuda, aw, nx, ny, Lx, Ly, 16, aw.AW_MODEL_DARWIN, dt=0.05)
    try:
        rng = np.random.default_rng(nx + ny)
        src = {k: rng.normal(0, 1, (ny, nx)).astype(np.float32) for k in ("rho", "Jx", "Jy", "Jz")}
        for k, v in src.items():
            s.put(k, v)
        s.ctx.solve_darwin_el_b()
        want = solve64(nx, ny, (Lx, Ly), src["rho"].astype(float), [src[k].astype(float) for k in ("Jx", "Jy", "Jz")])
        for k, w in zip(("ELx", "ELy", "Bx", "By", "Bz"), want):
            got = s.grid(k)
            assert np.abs(got - w).max() <= 2e-6 * np.abs(w).max(), k
    finally:
        s.close()


# every solve on the path these grids take: both longest sides (seven planes of a column
# of 1024 in shared memory), odd sides, every radix
ALL_SHAPES = [(64, 64), (75, 63), (98, 54), (48, 1024), (1024, 50), (105, 49)]


def rel2(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("nx,ny", ALL_SHAPES)
@pytest.mark.parametrize("smooth", [dict(), dict(ax=0.3, ay=0.2, cic_order=1, k_filter=9.0)])
def test_every_solve_matches_fp64(torch_cuda, aw, nx, ny, smooth):
    """E from rho, E_L and B, E_T, each with and without a form factor (its table is
    read in the order of the transposed planes)."""
    from oracle import formfactor64 as ff
    Lx, Ly = 0.3 * nx, 0.2 * ny
    s = Setup(torch_cuda, aw, nx, ny, Lx, Ly, 16, aw.AW_MODEL_DARWIN, dt=0.05)
    try:
        rng = np.random.default_rng(7 * nx + ny)
        names = ("rho", "Jx", "Jy", "Jz", "dcux", "dcuy", "dcuz", "amu0", "amu1", "amu2", "amu3")
        src = {k: rng.normal(0, 1, (ny, nx)).astype(np.float32) for k in names}
        for k, v in src.items():
            s.put(k, v)
        if smooth:
            s.ctx.set_form_factor(**smooth)
        sm = ff.form_factor(nx, ny, Lx, Ly, **smooth)
        d = {k: v.astype(float) for k, v in src.items()}
        s.ctx.solve_es()
        s.ctx.solve_darwin_el_b()
        s.ctx.solve_darwin_et()
        want = dict(zip(("Ex", "Ey"), ff.solve_es(d["rho"], Lx, Ly, sm)))
        want.update(zip(("ELx", "ELy", "Bx", "By", "Bz"), ff.solve_elb(*(d[k] for k in names[:4]), Lx, Ly, sm)))
        want.update(zip(("ETx", "ETy", "ETz"), ff.solve_et(np.stack([d[k] for k in names[4:7]]),
                                                           np.stack([d[k] for k in names[7:]]), Lx, Ly, sm)))
        for k, w in want.items():
            got = s.grid(k)
            assert rel2(got, w) < 1e-6, k
            assert np.abs(got - w).max() <= 2e-6 * np.abs(w).max(), k
    finally:
        s.close()


@pytest.mark.parametrize("nx,ny", [(128, 128), (375, 225), (1024, 128), (720, 96), (63, 64)])
def test_a_planes_mean_adds_no_error(torch_cuda, aw, nx, ny):
    """Sources whose mean is twenty times their spread (a charge density's, a drifting
    plasma's current): the k = 0 mode is not used, and its roundoff, 2^-24 x 20 per
    element, stays out of the others. Ten roundings of 2^-24: 6e-7."""
    from oracle import formfactor64 as ff
    Lx, Ly = 0.5 * nx, 0.5 * ny
    s = Setup(torch_cuda, aw, nx, ny, Lx, Ly, 16, aw.AW_MODEL_DARWIN, dt=0.05)
    try:
        rng = np.random.default_rng(nx)
        src = {k: rng.normal(m, 1, (ny, nx)).astype(np.float32) for k, m in (("rho", -20), ("Jx", 20), ("Jy", -20), ("Jz", 20))}
        for k, v in src.items():
            s.put(k, v)
        s.ctx.solve_darwin_el_b()
        one = np.ones((ny, nx // 2 + 1))
        want = ff.solve_elb(*(src[k].astype(float) for k in ("rho", "Jx", "Jy", "Jz")), Lx, Ly, one)
        for k, w in zip(("ELx", "ELy", "Bx", "By", "Bz"), want):
            assert rel2(s.grid(k), w) < 6e-7, (k, rel2(s.grid(k), w))
    finally:
        s.close()


@pytest.mark.parametrize("nx,ny", [(720, 96), (96, 720), (375, 225), (64, 60), (400, 64), (625, 48), (343, 64)])
def test_no_further_from_fp64_than_the_library_transforms(torch_cuda, aw, nx, ny):
    """White sources: the error against 64 bits is no larger than that of the same solve
    through the library's single precision transforms."""
    torch = torch_cuda
    Lx, Ly = 0.5 * nx, 0.5 * ny
    s = Setup(torch, aw, nx, ny, Lx, Ly, 16, aw.AW_MODEL_DARWIN, dt=0.05)
    try:
        g = torch.Generator(device=s.dev)
        g.manual_seed(nx + ny)
        kx = torch.arange(nx // 2 + 1, device=s.dev, dtype=torch.float64) * (2 * np.pi / Lx)
        m = torch.arange(ny, device=s.dev, dtype=torch.float64)
        ky = (torch.where(m <= ny // 2, m, m - ny) * (2 * np.pi / Ly))[:, None]
        k2 = kx * kx + ky * ky
        keep = (k2 > 0).double()
        if nx % 2 == 0:
            keep[:, nx // 2] = 0
        if ny % 2 == 0:
            keep[ny // 2] = 0
        green = keep / torch.where(k2 > 0, k2, torch.ones_like(k2))
        ours = theirs = 0.0
        for _ in range(4):
            for k in ("rho", "Jx", "Jy", "Jz"):
                s.G[k].normal_(generator=g)
            s.ctx.solve_darwin_el_b()
            torch.cuda.synchronize()
            src = {k: s.G[k].reshape(ny, nx) for k in ("rho", "Jx", "Jy", "Jz")}
            F, f = ({k: torch.fft.rfft2(v.to(t)) for k, v in src.items()} for t in (torch.float64, torch.float32))
            mul = {"ELx": (("rho", -1j * kx * green),), "Bx": (("Jz", 1j * ky * green),),
                   "Bz": (("Jy", 1j * kx * green), ("Jx", -1j * ky * green))}
            for k, terms in mul.items():
                want = torch.fft.irfft2(sum(F[q] * c for q, c in terms), s=(ny, nx))
                lib = torch.fft.irfft2(sum(f[q].to(torch.complex128) * c for q, c in terms).to(torch.complex64), s=(ny, nx))
                e = lambda a: float((a.double() - want).square().sum() / want.square().sum())  # noqa: E731
                ours += e(s.G[k].reshape(ny, nx))
                theirs += e(lib)
        assert ours <= theirs, (ours ** 0.5, theirs ** 0.5)
    finally:
        s.close()


@pytest.mark.parametrize("nx,ny,smooth", [(48, 48, dict()), (50, 63, dict()), (60, 56, dict(ax=0.7, ay=0.4, cic_order=1))])
def test_es_gradient_matches_fp64(torch_cuda, aw, nx, ny, smooth):
    """aw_grad_es on grids whose transposed solve takes this path, with the bars of
    test_gpu_adjoint.py."""
    from gpu_helpers import TWO_STREAM, n_particles
    from oracle.adjoint64 import Case
    from oracle.formfactor64 import form_factor
    nsteps = 12
    s = Setup(torch_cuda, aw, nx, ny, float(nx), float(ny), n_particles(TWO_STREAM, nx, ny), aw.AW_MODEL_ES, dt=0.1,
              B0=(0.3, 0.1, 0.2))
    try:
        s.ctx.load_species(TWO_STREAM, seed=1, noisy=True)
        if smooth:
            s.ctx.set_form_factor(**smooth)
        p = s.parts()
        du = [torch_cuda.zeros(s.n, dtype=torch_cuda.float32, device=s.dev) for _ in range(3)]
        loss = s.ctx.grad_es(nsteps, 5, *du)
        g = np.stack([d.cpu().numpy().astype(float) for d in du], axis=1)
        sm = form_factor(nx, ny, float(nx), float(ny), **smooth) if smooth else None
        case = Case(nx, ny, float(nx), float(ny), 0.1, B0=(0.3, 0.1, 0.2), smooth=sm)
        u0 = np.stack([p[k] for k in ("ux", "uy", "uz")], axis=1).astype(float)
        L64, g64 = case.gradient(p["x"].astype(float), p["y"].astype(float), u0, p["w"].astype(float), nsteps)
        assert abs(loss - L64) <= 1e-4 * abs(L64), (loss, L64)
        assert rel2(g, g64) < 2e-3, rel2(g, g64)
    finally:
        s.close()


@pytest.mark.parametrize("nx,ny", [(48, 48), (50, 63)])
def test_darwin_gradient_matches_fp64(torch_cuda, aw, nx, ny):
    """aw_grad_darwin likewise: the transposes of both Darwin solves."""
    from oracle.darwin_adjoint64 import DarwinCase
    sp = [dict(ppc=8, density=1.0, uth=(0.05, 0.05, 0.2), ufl=(0.0, 0.0, 0.0))]
    B0, Lx, Ly, nsteps = (0.3, 0.2, 0.4), 0.5 * nx, 0.5 * ny, 6
    pump = dict(ex=2e-2, ey=3e-2, ez=-1e-2, k0=2 * np.pi * 2 / Lx, w0=0.3, trmp=0.2, toff=100.0)
    s = Setup(torch_cuda, aw, nx, ny, Lx, Ly, 8 * nx * ny, aw.AW_MODEL_DARWIN, dt=0.05, B0=B0, pump=pump)
    try:
        s.ctx.load_species(sp, seed=3, noisy=True)
        p = s.parts()
        du = [torch_cuda.zeros(s.n, dtype=torch_cuda.float32, device=s.dev) for _ in range(3)]
        loss, dpump = s.ctx.grad_darwin(nsteps, 4, *du)
        g = np.stack([d.cpu().numpy().astype(float) for d in du], axis=1)
        assert s.ctx.error_word() == 0
        case = DarwinCase(nx, ny, Lx, Ly, 0.05, B0=B0, pump=pump)
        u0 = np.stack([p[k] for k in ("ux", "uy", "uz")], axis=1).astype(float)
        L64, g64, dp64 = case.gradient(p["x"].astype(float), p["y"].astype(float), u0, p["w"].astype(float), nsteps)
        assert abs(loss - L64) <= 1e-5 * abs(L64), (loss, L64)
        assert rel2(g, g64) < 5e-5, rel2(g, g64)
        assert abs(dpump - dp64) <= 1e-4 * abs(dp64), (dpump, dp64)
    finally:
        s.close()
