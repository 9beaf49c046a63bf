"""aw_ensemble_*: independent runs advanced together by one graph launch per
step. Every run equals the same run done alone, bit for bit (diagnostics and
particle state), whether the ensemble runs concurrently or one run after
another; the autotuner's choices do not change any result."""
import numpy as np
import pytest

from gpu_helpers import PARTICLE_KEYS, d2h

pytestmark = pytest.mark.gpu

SIDES, PPCS = (16, 32, 64), (4, 16)


def _alone(torch, aw, d, nsteps):
    """The run of draw d on its own context (the reference's one-Simulation way)."""
    from arcwarden_b200.ensemble import spec_of
    sp = spec_of(d)
    n = d["side"] * d["side"] * d["ppc"]
    dev = torch.device("cuda:0")
    P = {k: torch.zeros(n, dtype=torch.float32, device=dev) for k in PARTICLE_KEYS}
    cell = torch.zeros(n, dtype=torch.int32, device=dev)
    ctx = aw.Context(d["side"], d["side"], float(d["side"]), float(d["side"]), model=sp.model, dt=sp.params.dt,
                     c=1.0, n0=1.0, B0=d["B0"], stream=torch.cuda.current_stream().cuda_stream)
    try:
        ctx.bind_particles(*(P[k] for k in PARTICLE_KEYS), cell)
        half = d["ppc"] // 2
        ctx.load_species([dict(ppc=half, density=0.5, uth=(d["vth"],) * 3, ufl=(d["vd"], 0.0, 0.0)),
                          dict(ppc=d["ppc"] - half, density=0.5, uth=(d["vth"],) * 3, ufl=(-d["vd"], 0.0, 0.0))],
                         seed=d["seed"], noisy=True)
        ctx.init()
        ctx.run(0, nsteps, graph=True)
        torch.cuda.synchronize()
        return ctx.step_diag(), {k: P[k].cpu().numpy() for k in ("x", "y", "ux", "uy", "uz")}
    finally:
        ctx.close()


def _ens_state(torch, e, run, keys=("x", "y", "ux", "uy", "uz")):
    ptrs, n = e.particles(run)
    return {k: d2h(torch, ptrs[k], n, np.float32) for k in keys}


@pytest.mark.parametrize("concurrent, sides, nruns", [
    (True, SIDES, 8), (False, SIDES, 8),
    (True, (32, 256), 6),          # 256^2 x 16 ppc: 512 chunks, a run with its own step graph
])
def test_ensemble_runs_equal_runs_alone(torch_cuda, aw, concurrent, sides, nruns):
    from arcwarden_b200.ensemble import ensemble_specs
    draws, specs = ensemble_specs(nruns, sides, (16,) if sides != SIDES else PPCS)
    e = aw.Ensemble(specs)
    try:
        e.init()
        e.run(4, concurrent=concurrent)
        e.run(3, concurrent=concurrent)
        torch_cuda.cuda.synchronize()
        for r, d in enumerate(draws):
            diag, state = _alone(torch_cuda, aw, d, 7)
            assert e.diag(r) == diag, r
            got = _ens_state(torch_cuda, e, r)
            for k in state:
                assert np.array_equal(got[k], state[k]), (r, k)
    finally:
        e.close()


def test_ensemble_autotuner_keeps_results(torch_cuda, aw):
    from arcwarden_b200.ensemble import ensemble_specs
    draws, specs = ensemble_specs(6, SIDES, PPCS)
    a, b = aw.Ensemble(specs), aw.Ensemble(specs)
    try:
        b.tune(3)
        for r in range(len(specs)):
            every, tile = b.tuning(r)
            assert every in (0, 50) and tile in (512, 1024, 2048)
        a.init()
        b.init()
        a.run(60)
        b.run(60)
        torch_cuda.cuda.synchronize()
        for r in range(len(specs)):
            da, db = a.diag(r), b.diag(r)
            # the re-sort permutes particles only and the deposit is order-free; the
            # per-chunk partial sums (KE, momentum, the coefficient rms behind the
            # Darwin J/amu scales) see different chunks, so the last bits may move
            assert da["charge"] == db["charge"], r
            for k in ("ee", "max_e", "eb", "ke", "px", "py", "pz"):
                assert abs(da[k] - db[k]) <= 1e-6 * max(1e-9, abs(da[k])), (r, k, da[k], db[k])
    finally:
        a.close()
        b.close()


def test_ensemble_rejects_bad_specs(aw):
    from arcwarden_b200.ensemble import ensemble_specs
    _, specs = ensemble_specs(1, SIDES, PPCS)
    specs[0].nspecies = 0
    with pytest.raises(aw.ArcError):
        aw.Ensemble(specs)


@pytest.mark.parametrize("model", [0, 1])
def test_members_of_every_chunk_size_equal_runs_alone(torch_cuda, aw, model):
    """A run alone takes chunks of 256 to 2048 particles, by its own size; in an ensemble
    the particle kernels take full ones and the sums go over the run's own: the same
    bits in the state and the diagnostics, ragged counts and odd grids included, for
    runs that share launches and runs with their own step."""
    #        nx   ny  per beam
    runs = [(50, 30, 5), (64, 64, 8), (64, 64, 33), (75, 64, 27), (128, 96, 21), (128, 64, 45), (256, 130, 16)]
    beams = lambda ppc: [dict(ppc=ppc, density=0.5, uth=(0.05, 0.04, 0.06), ufl=(v, 0.02, 0.0)) for v in (0.2, -0.25)]  # noqa: E731
    par = dict(dt=0.05, c=1.0, n0=1.0, B0=(0.1, 0.0, 0.4))
    e = aw.Ensemble([aw.run_spec(model, nx, ny, float(nx), float(ny), beams(p), seed=k, **par)
                     for k, (nx, ny, p) in enumerate(runs)])
    try:
        e.init()
        e.run(3)
        e.run(2)
        torch_cuda.cuda.synchronize()
        for k, (nx, ny, p) in enumerate(runs):
            n = 2 * p * nx * ny
            P = {q: torch_cuda.zeros(n, dtype=torch_cuda.float32, device="cuda:0") for q in PARTICLE_KEYS}
            cell = torch_cuda.zeros(n, dtype=torch_cuda.int32, device="cuda:0")
            ctx = aw.Context(nx, ny, float(nx), float(ny), model=model,
                             stream=torch_cuda.cuda.current_stream().cuda_stream, **par)
            try:
                ctx.bind_particles(*(P[q] for q in PARTICLE_KEYS), cell)
                ctx.load_species(beams(p), seed=k, noisy=True)
                ctx.init()
                ctx.run(0, 5)
                torch_cuda.cuda.synchronize()
                assert ctx.error_word() == 0
                assert e.diag(k) == ctx.step_diag(), k
                got = _ens_state(torch_cuda, e, k)
                for q in got:
                    assert np.array_equal(got[q], P[q].cpu().numpy()), (k, q)
            finally:
                ctx.close()
    finally:
        e.close()
