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
