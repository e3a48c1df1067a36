"""The bins step on uniform centres (suffix scan) and on centres that are not
(FFT), against the oracle's direct long-double convolution and its tracking.

Tolerance of the potential: the scan's sums run over non-negative densities with
factors of modulus below one, so with S = Σg and A the wake's amplitude each
suffix sum carries at most about 4 eps (E + 5 + log2(warps) + CTAs) <= 104 eps of
S, a power of σ at most 14 products of 3 eps, and two such terms enter a
potential: below 300 eps |A| S = 3.4e-14 |A| S.  1e-13 of |current A| S is asked."""
import numpy as np
import pytest
import torch

from haissinskijulia_b200 import BinGrid, ResidentBunch, WakeModel, benchmark_ring
from oracle import pyoracle

from gpu_util import assert_close, device_pair

pytestmark = pytest.mark.gpu

N = 20_011
TURNS = 2


def _wake(kind):
    w = benchmark_ring().wake
    if kind == "short":          # decays within a bin or two
        return WakeModel(w.wake_factor, w.wake_sqrt, 1e-6, w.sin_coef, 1e9, 6.0)
    if kind == "long":           # no decay over the grid
        return WakeModel(1e-3 * w.wake_factor, 40.0, 1e3, 0.0, 1e9, 6.0)
    if kind == "reference":      # no sine term, the reference's constants
        return WakeModel(3.6e14, 490.0, 4e-3, 0.0, 1e9, 7.5)
    return w


def _grid(sigma_z, nbins, kind):
    g = BinGrid.make(sigma_z, nbins, 6.0)
    if kind == "uniform":
        return g
    h = g.edge_step
    if kind.startswith("jittered"):       # ordered, not uniform
        c = g.centers + 0.2 * h * np.sin(1.7 * np.arange(nbins))
        if kind == "jittered_inside":     # the interpolation's cells are those of the edges
            c[0], c[-1] = g.centers[0], g.centers[-1]
        return BinGrid(g.edge_first, g.edge_last, h, c)
    # uniform, but bin 0's neighbourhood of z = 0 sits elsewhere in the grid
    off = {"low": -2.5, "high": 2.5, "all_below": -6.5, "all_above": 6.5}[kind] * sigma_z
    return BinGrid(g.edge_first + off, g.edge_last + off, h, g.centers + off)


def _run(gpu_ctx, oracle, nbins, wake_kind="resonator", grid_kind="uniform"):
    cfg = benchmark_ring(n_turns=TURNS, nbins=nbins)
    wake = _wake(wake_kind)
    rng = np.random.default_rng(nbins + len(wake_kind) + len(grid_kind))
    z0, e0 = rng.normal(0.0, cfg.sigma_z, N), rng.normal(0.0, cfg.sigma_E, N)
    draws = rng.normal(size=(TURNS, N))
    grid = _grid(oracle.global_std(z0), nbins, grid_kind)
    dz, de = device_pair(z0, e0)
    dd = torch.from_numpy(draws).cuda()
    b = ResidentBunch(gpu_ctx, dz.data_ptr(), de.data_ptr(), N, cfg.params, nbins, wake=wake,
                      grid=grid, seed=3)
    b.set_draws(dd.data_ptr(), 1, TURNS)
    zo, eo = z0.copy(), e0.copy()
    st = oracle.state(zo, eo, cfg.params.to_c(), wake.to_c(), nbins, grid.to_c())
    zout, eout = torch.empty_like(dz), torch.empty_like(de)
    for t in range(TURNS):
        b.advance(1)
        assert st.turn(np.ascontiguousarray(draws[t])) == 0
        r = b.observe(zout.data_ptr(), eout.data_ptr())
        counts = b.histogram()
        assert np.array_equal(counts, st.counts())
        exact = oracle.wake_potential(counts, grid.to_c(), wake.to_c(), st.last_current,
                                      pyoracle.CONV_DIRECT_LD)
        lam = np.exp(-0.5 * (grid.centers / wake.delta_std) ** 2) / (
            np.sqrt(2 * np.pi) * wake.delta_std)
        dens = lam * counts / max(1, counts.sum())
        amp = abs(wake.wake_factor) * np.hypot(1.0, wake.sin_coef)
        full = abs(st.last_current) * amp * dens.sum()
        assert np.abs(b.potential() - exact).max() <= 1e-13 * full, t
        if grid_kind == "jittered":
            break       # the pass takes its kick cells from the edges: these centres move them
        assert_close(zout.cpu().numpy(), zo, cfg.sigma_z, what=f"z turn {t}")
        assert_close(eout.cpu().numpy(), eo, cfg.sigma_E, what=f"dE turn {t}")
        assert abs(r.E0 - st.E0) <= 1e-12 * st.E0
    b.close()


@pytest.mark.parametrize("nbins", [1, 2, 3, 7, 255, 256, 511, 512, 513, 1023, 1024, 1025, 2047,
                                   2048, 2049, 4095, 4096, 4097, 8191, 8192, 8193, 16383, 16384])
def test_scan_at_the_edges_of_its_forms(gpu_ctx, oracle, nbins):
    _run(gpu_ctx, oracle, nbins)


@pytest.mark.parametrize("wake_kind", ["short", "long", "reference"])
@pytest.mark.parametrize("nbins", [777, 4096])
def test_scan_of_other_wakes(gpu_ctx, oracle, wake_kind, nbins):
    _run(gpu_ctx, oracle, nbins, wake_kind)


@pytest.mark.parametrize("grid_kind", ["low", "high", "all_below", "all_above", "jittered",
                                       "jittered_inside"])
@pytest.mark.parametrize("nbins", [5, 1000, 4096, 10000])
def test_other_centres(gpu_ctx, oracle, grid_kind, nbins):
    _run(gpu_ctx, oracle, nbins, grid_kind=grid_kind)
