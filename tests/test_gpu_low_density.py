"""The electrostatic push's two-pass fallback at few particles per cell, where a chunk
is whole grid rows and their spread: the window asked for is the window taken, the
built-in one holds what such chunks cover, and no choice changes a result."""
import numpy as np
import pytest

from gpu_helpers import PARTICLE_KEYS, Setup

pytestmark = pytest.mark.gpu


def spread_rows(nx, ny, ppc, rows, seed=5):
    """Particles in cell order, moved up to `rows` rows and columns from their cell."""
    n = nx * ny * ppc
    rng = np.random.default_rng(seed)
    cell = np.repeat(np.arange(nx * ny), ppc)
    x = (cell % nx + rng.uniform(-rows, rows, n)) % nx
    y = (cell // nx + rng.uniform(-rows, rows, n)) % ny
    top = lambda v, m: np.minimum(v.astype(np.float32), np.nextafter(np.float32(m), np.float32(0)))  # noqa: E731
    return {"x": top(x, nx), "y": top(y, ny), "ux": rng.normal(0, 0.05, n), "uy": rng.normal(0, 0.05, n),
            "uz": rng.normal(0, 0.05, n), "w": np.full(n, 1.0 / ppc)}


def steps(torch, aw, nx, ny, ppc, rows, window, nsteps=3):
    P = spread_rows(nx, ny, ppc, rows)
    s = Setup(torch, aw, nx, ny, float(nx), float(ny), nx * ny * ppc, aw.AW_MODEL_ES, dt=0.05)
    try:
        s.ctx.set_kernel_plan(es_window=window)
        for k in PARTICLE_KEYS:
            s.put(k, P[k].astype(np.float32))
        s.ctx.init()
        before = s.ctx.stats()
        s.ctx.run(0, nsteps)
        st = s.ctx.stats()
        r = s.parts()
        for k in ("rho", "Ex", "Ey"):
            r[k] = s.grid(k)
        assert s.ctx.error_word() == 0
        return r, {k: st[k] - before[k] for k in ("chunks", "window_overflow", "slow_deposits")}
    finally:
        s.close()


@pytest.mark.parametrize("nx,ny,ppc,rows", [(256, 256, 8, 4), (500, 120, 8, 6)])
def test_window_capacity_is_the_one_asked_for(torch_cuda, aw, nx, ny, ppc, rows):
    """Boxes of up to 2313 (1960) cells: one band at 3584 and 4096 cells, several at 1024 (and
    the overflow counter counts a banded chunk); the same bits from every capacity."""
    out = {w: steps(torch_cuda, aw, nx, ny, ppc, rows, w) for w in (0, 256, 1024, 3584, 4096)}
    assert out[1024][1]["window_overflow"] > 0.9 * out[1024][1]["chunks"]
    assert out[3584][1]["window_overflow"] == 0 and out[4096][1]["window_overflow"] == 0
    assert out[0][1]["window_overflow"] == 0, "the built-in window at this density"
    for w in out:
        for k in out[0][0]:
            assert np.array_equal(out[w][0][k], out[0][0][k]), (w, k)
