"""A bunch whose particles all sit at one z has no length: the wake current, proportional
to σ_z (src/evolution.jl:357, :386), is exactly zero.  z = 2^-9 makes every sum exact; the
harmonic number 0 switches the drift off, so z stays.  (The oracle's drift goes through
the phase and back, which moves its z by a rounding and its current to 1e-19 or so.)"""
import numpy as np
import pytest

from haissinskijulia_b200 import BinGrid, ResidentBunch, benchmark_ring, gaussian_draws

from gpu_util import assert_close, device_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nbins", [64, 4096])
@pytest.mark.parametrize("n", [2, 5, 49, 66, 1000, 20_011])
def test_no_length_no_wake(gpu_ctx, gpu_buffers, oracle, n, nbins):
    cfg = benchmark_ring(n_turns=2, nbins=nbins)
    cfg.params.harmonic = 0
    z = np.full(n, 2.0 ** -9)
    e = np.where(np.arange(n) % 2 == 0, 1e5, -1e5).astype(np.float64)
    grid = BinGrid.make(1e-3, nbins, 6.0)
    dz, de = device_pair(z, e)
    b = ResidentBunch(gpu_ctx, dz.data_ptr(), de.data_ptr(), n, cfg.params, nbins, wake=cfg.wake,
                      grid=grid, seed=4)
    b.set_log(1, capacity=4)
    st = oracle.state(z, e, cfg.params.to_c(), cfg.wake.to_c(), nbins, grid.to_c())
    for t in (1, 2):
        b.advance(1)
        assert st.turn(np.ascontiguousarray(gaussian_draws(4, t, n, gpu_buffers))) == 0
    assert (b.read_log()[:, 6] == 0.0).all()
    assert (b.potential() == 0.0).all()
    b.finish()
    assert np.array_equal(dz.cpu().numpy(), np.full(n, 2.0 ** -9))
    assert_close(de.cpu().numpy(), e, cfg.sigma_E, what="dE")
    b.close()
    st.close()
