"""Particles into and out of a batch by the moments kernel (device memory, any
8-byte alignment) against the copies of the host path, and the pass at sizes
around whole warps of four-particle groups against the oracle.

The device and host routes run the same kernels on the same particles, so they must
agree bit for bit; against the oracle the suite's 1e-12 relative holds."""
import numpy as np
import pytest
import torch

from haissinskijulia_b200 import Batch, BinGrid, ResidentBunch, benchmark_ring, gaussian_draws

from gpu_util import assert_close, device_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 2047, 2048, 2051, 40_003])
def test_device_memory_takes_the_host_routes_values(gpu_ctx, n, shift):
    cfg = benchmark_ring(n_turns=1, nbins=256)
    rng = np.random.default_rng(n)
    z, e = rng.normal(0.0, cfg.sigma_z, n), rng.normal(0.0, cfg.sigma_E, n)
    for turns in (0, 3):
        if n < 2 and turns:
            continue                      # one particle has no spread for the wake
        bt = Batch(gpu_ctx, 2 * (n + 8), 2, 256)
        pad = torch.zeros(4, n + 8, dtype=torch.float64, device="cuda")
        src = pad[:2, shift:shift + n]
        src.copy_(torch.from_numpy(np.stack([z, e])))
        torch.cuda.synchronize()
        a = bt.add_device(src[0].data_ptr(), src[1].data_ptr(), n, cfg.params, 256, wake=cfg.wake,
                          seed=5, turns=turns)
        b = bt.add(z, e, cfg.params, 256, wake=cfg.wake, seed=5, turns=turns)
        if turns:
            bt.advance(turns)
        assert sorted(bt.poll()) == sorted([a, b])
        out = pad[2:, shift:shift + n]
        ra = bt.take_device(a, out[0].data_ptr(), out[1].data_ptr())
        zb, eb, rb = bt.take(b)
        za, ea = out.cpu().numpy()
        assert np.array_equal(za, zb) and np.array_equal(ea, eb)
        assert ra == rb
        if turns == 0:
            assert np.array_equal(za, z) and np.array_equal(ea, e)
        rest = pad.cpu().numpy()
        rest[:, shift:shift + n] = 0.0
        assert not rest.any()             # nothing outside the slices was written
        bt.close()


@pytest.mark.parametrize("n", [2, 5, 127, 128, 129, 511, 515, 2048, 2175, 2176, 16_511])
def test_pass_around_whole_warps(gpu_ctx, gpu_buffers, oracle, n):
    turns, nbins = 3, 512
    cfg = benchmark_ring(n_turns=turns, nbins=nbins)
    rng = np.random.default_rng(n)
    z, e = rng.normal(0.0, cfg.sigma_z, n), rng.normal(0.0, cfg.sigma_E, n)
    grid = BinGrid.make(cfg.sigma_z, nbins, 6.0)
    dz, de = device_pair(z, e)
    b = ResidentBunch(gpu_ctx, dz.data_ptr(), de.data_ptr(), n, cfg.params, nbins, wake=cfg.wake,
                      grid=grid, seed=9)
    st = oracle.state(z, e, cfg.params.to_c(), cfg.wake.to_c(), nbins, grid.to_c())
    for t in range(1, turns + 1):
        b.advance(1)
        assert st.turn(np.ascontiguousarray(gaussian_draws(9, t, n, gpu_buffers))) == 0
        assert np.array_equal(b.histogram(), st.counts()), t
    b.finish()
    assert_close(dz.cpu().numpy(), z, cfg.sigma_z, what="z")
    assert_close(de.cpu().numpy(), e, cfg.sigma_E, what="dE")
    b.close()
