"""aw_run_diag over more steps than the device's record ring holds (1024): the batches'
records, the re-sorts that fall between and inside them and the state after them are
those of shorter calls."""
import numpy as np
import pytest

from gpu_helpers import PARTICLE_KEYS, TWO_STREAM, WEIBEL, Setup, n_particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,species,nsteps,pieces", [
    (0, TWO_STREAM, 2100, (1, 1023, 1024, 52)),
    (1, WEIBEL, 1100, (1000, 100))])
def test_batches_of_the_ring_equal_shorter_calls(torch_cuda, aw, model, species, nsteps, pieces):
    assert sum(pieces) == nsteps
    out = []
    for cut in ((nsteps,), pieces):
        s = Setup(torch_cuda, aw, 16, 16, 16.0, 16.0, n_particles(species, 16, 16), model, dt=0.05)
        try:
            s.ctx.load_species(species, seed=9, noisy=True)
            s.ctx.init()
            d = np.zeros((nsteps + 1, 8))
            at = 0
            for m in cut:
                s.ctx.run_diag(at, m, d[at:].ctypes.data)
                at += m
            torch_cuda.cuda.synchronize()
            assert s.ctx.error_word() == 0
            assert not d[nsteps].any() and (d[:nsteps, 0] > 0).all()      # every record, and not one more
            assert dict(zip(s.ctx.step_diag(), d[nsteps - 1])) == s.ctx.step_diag()
            out.append((d, s.parts()))
        finally:
            s.close()
    assert np.array_equal(out[0][0], out[1][0])
    for k in PARTICLE_KEYS:
        assert np.array_equal(out[0][1][k], out[1][1][k]), k
