"""Caller's grids whose histogram bins (between the edges) and interpolation cells
(between the centres) do not fit together half a bin apart: the histogram follows the
edges and the kick the centres (src/utils.jl:387-397, src/wakefield.jl:64-102), against
the oracle turn by turn.

Counts are integers and must agree; particles within the suite's 1e-12 relative."""
import numpy as np
import pytest
import torch

from haissinskijulia_b200 import BinGrid, Context, ResidentBunch, benchmark_ring, gaussian_draws

from gpu_util import assert_close, device_pair

pytestmark = pytest.mark.gpu

N = 30_011
TURNS = 3
KINDS = ["shifted", "moved_ends", "narrow_edges", "coarse_edges", "short_last", "descending",
         "no_bin"]


def _grid(sigma_z, nbins, kind):
    g = BinGrid.make(sigma_z, nbins, 6.0)
    h, c = g.edge_step, np.array(g.centers)
    if kind == "shifted":                       # uniform, 0.3 bins off the edges
        return BinGrid(g.edge_first, g.edge_last, h, c + 0.3 * h)
    if kind == "moved_ends":                    # neither uniform nor at the midpoints
        c = c + 0.2 * h * np.sin(1.7 * np.arange(nbins) + 1.0)
        return BinGrid(g.edge_first, g.edge_last, h, c)
    if kind == "narrow_edges":                  # bins over half of the centres' range
        return BinGrid(0.5 * g.edge_first, 0.5 * g.edge_last, 0.5 * h, c)
    if kind == "coarse_edges":                  # and over more than it
        return BinGrid(1.3 * g.edge_first, 1.3 * g.edge_last, 1.3 * h, c)
    if kind == "short_last":                    # the last edge cuts bins off
        return BinGrid(g.edge_first, g.edge_last - 0.3 * (g.edge_last - g.edge_first), h, c)
    if kind == "descending":                    # clamp(z, c1, cB) is cB for every z
        return BinGrid(g.edge_first, g.edge_last, h, c[::-1].copy())
    return BinGrid(g.edge_last, g.edge_first, -h, c)    # no z lies between the edges


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("nbins", [1, 2, 5, 1000, 4097, 16384])
@pytest.mark.parametrize("normals", ["float64", "draws"])
def test_split_grid_against_the_oracle(gpu_buffers, oracle, kind, nbins, normals):
    cfg = benchmark_ring(n_turns=TURNS, nbins=nbins)
    rng = np.random.default_rng(nbins + len(kind))
    z, e = rng.normal(0.0, cfg.sigma_z, N), rng.normal(0.0, cfg.sigma_E, N)
    grid = _grid(oracle.global_std(z), nbins, kind)
    ctx = Context(0)
    if normals == "draws":
        ctx.set_pass_layout(1)                  # the layout is the library's for such grids
    dz, de = device_pair(z, e)
    b = ResidentBunch(ctx, dz.data_ptr(), de.data_ptr(), N, cfg.params, nbins, wake=cfg.wake,
                      grid=grid, seed=23)
    if normals == "draws":
        draws = rng.normal(size=(TURNS, N))
        dd = torch.from_numpy(draws).cuda()
        b.set_draws(dd.data_ptr(), 1, TURNS)
    else:
        draws = [gaussian_draws(23, t, N, gpu_buffers) for t in range(1, TURNS + 1)]
    st = oracle.state(z, e, cfg.params.to_c(), cfg.wake.to_c(), nbins, grid.to_c())
    zout, eout = torch.empty_like(dz), torch.empty_like(de)
    for t in range(TURNS):
        b.advance(1)
        assert st.turn(np.ascontiguousarray(draws[t])) == 0
        r = b.observe(zout.data_ptr(), eout.data_ptr())
        assert np.array_equal(b.histogram(), st.counts()), t
        assert_close(zout.cpu().numpy(), z, cfg.sigma_z, what=f"z turn {t}")
        assert_close(eout.cpu().numpy(), e, cfg.sigma_E, what=f"dE turn {t}")
        assert abs(r.E0 - st.E0) <= 1e-12 * st.E0
    b.close()
    st.close()
    ctx.close()
