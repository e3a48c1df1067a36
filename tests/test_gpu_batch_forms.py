"""Every form of the batched bins step (clusters by the batch's slots and largest bin count)
and every kind of block split, against the oracle: batches of 8 to 256 slots, members with
as many bins as the batch allows and fewer, blocks of 16384 to 131072 particles by the
default rule, and callers' own blocks on and off whole warps.

Counts are integers and must agree; particles within the suite's 1e-12 relative."""
import numpy as np
import pytest

from haissinskijulia_b200 import Batch, BinGrid, benchmark_ring, gaussian_draws

from gpu_util import assert_close

pytestmark = pytest.mark.gpu

TURNS = 3


def _run(gpu_ctx, gpu_buffers, oracle, slots, max_nbins, members, chunk=65536, resident=False):
    """members: (particles, bins) rows; the others of the slots stay free."""
    bt = Batch(gpu_ctx, sum(n + 4 for n, _ in members), slots, max_nbins, chunk=chunk,
               graph_turns=2, resident=resident)
    rows = []
    for i, (n, nbins) in enumerate(members):
        cfg = benchmark_ring(n_turns=TURNS, nbins=nbins, population=2e10 * (i + 1))
        rng = np.random.default_rng(100 * slots + i)
        z, e = rng.normal(0.0, cfg.sigma_z, n), rng.normal(0.0, cfg.sigma_E, n)
        bid = bt.add(z, e, cfg.params, nbins, wake=cfg.wake, seed=50 + i, turns=TURNS)
        rows.append((bid, z, e, cfg, nbins, 50 + i))
    bt.advance(TURNS)
    assert sorted(bt.poll()) == sorted(r[0] for r in rows)
    for bid, z, e, cfg, nbins, seed in rows:
        counts = bt.histogram(bid, nbins)
        zg, eg, res = bt.take(bid)
        grid = BinGrid.make(res.sigma_z0_initial, nbins, cfg.wake.half_width_sigmas)
        st = oracle.state(z, e, cfg.params.to_c(), cfg.wake.to_c(), nbins, grid.to_c())
        for t in range(1, TURNS + 1):
            draws = gaussian_draws(seed, t, z.size, gpu_buffers)
            assert st.turn(np.ascontiguousarray(draws)) == 0
        assert np.array_equal(counts, st.counts())
        assert_close(zg, z, cfg.sigma_z, what=f"z of {z.size} with {nbins} bins")
        assert_close(eg, e, cfg.sigma_E, what=f"dE of {z.size} with {nbins} bins")
        assert abs(res.E0 - st.E0) <= 1e-12 * st.E0
        st.close()
    bt.close()


@pytest.mark.parametrize("slots", [8, 16, 32, 64, 100, 256])
@pytest.mark.parametrize("max_nbins", [512, 1024, 2048, 4096, 8192, 16384])
def test_bins_step_forms(gpu_ctx, gpu_buffers, oracle, slots, max_nbins):
    _run(gpu_ctx, gpu_buffers, oracle, slots, max_nbins,
         [(6_011, max_nbins), (5_000, max_nbins // 2 + 1), (20_483, max_nbins - 3), (300, 77)])


@pytest.mark.parametrize("slots,n", [(256, 1_050_001), (256, 500_003), (32, 640_129), (2, 40_000)])
def test_default_blocks(gpu_ctx, gpu_buffers, oracle, slots, n):
    _run(gpu_ctx, gpu_buffers, oracle, slots, 4096, [(n, 4096), (4_097, 1000)])


@pytest.mark.parametrize("resident", [False, True])
@pytest.mark.parametrize("chunk", [4, 100, 4096, 54_056, 262_144, 2**20 - 8])
def test_callers_blocks(gpu_ctx, gpu_buffers, oracle, chunk, resident):
    n = {4: 1_003, 100: 20_003}.get(chunk, 270_001)
    _run(gpu_ctx, gpu_buffers, oracle, 4, 2048, [(n, 2048), (n // 3, 1500)], chunk, resident)
