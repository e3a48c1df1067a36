"""The host's rule for a caller's grid (csrc/hj_host.cpp): whether the interpolation
cells halve the histogram's bins to rounding, and the cell coordinate they are read
with, on the CPU."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from haissinskijulia_b200 import BinGrid

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "haissinskijulia_b200", "csrc")
DRIVER = r"""
#include <cstdio>
#include <vector>
#include "hj_host.h"
int main() {
  long long B;
  double e0, eN, h;
  while (scanf("%lld %la %la %la", &B, &e0, &eN, &h) == 4) {
    std::vector<double> c(B);
    for (auto& v : c) if (scanf("%la", &v) != 1) return 1;
    hj_grid g{B, e0, eN, h, c.data()};
    const bool halves = hj::host_cells_halve_bins(g);
    const double step = B > 1 ? (c[B - 1] - c[0]) / (double)(B - 1) : 1.0;
    double inv, off;
    hj::host_kick_cells(halves, B, e0, 1.0 / h, c[0], c[B - 1], 1.0 / step, &inv, &off);
    printf("%d %a %a\n", halves ? 1 : 0, inv, off);
  }
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("kick")
    (d / "k.cpp").write_text(DRIVER)
    exe = str(d / "k")
    subprocess.run([gxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I", CSRC, str(d / "k.cpp"),
                    os.path.join(CSRC, "hj_host.cpp"), "-o", exe], check=True)

    def run(e0, eN, h, c):
        text = " ".join([str(len(c))] + [float(v).hex() for v in (e0, eN, h, *c)])
        out = subprocess.run([exe], input=text, capture_output=True, text=True,
                             check=True).stdout.split()
        return out[0] == "1", float.fromhex(out[1]), float.fromhex(out[2])
    return run


@pytest.mark.parametrize("nbins", [1, 2, 3, 100, 4096, 10007, 16384])
@pytest.mark.parametrize("sigma", [3.7e-3, 1e-12, 2.5])
def test_grids_of_the_library_and_of_linspace_halve(rule, nbins, sigma):
    g = BinGrid.make(sigma, nbins, 7.5)
    assert rule(g.edge_first, g.edge_last, g.edge_step, g.centers)[0]
    for off in (0.0, 3.0 * sigma):
        edges = np.linspace(-6 * sigma, 6 * sigma, nbins + 1) + off
        c = 0.5 * (edges[:-1] + edges[1:])
        assert rule(edges[0], edges[-1], (edges[-1] - edges[0]) / nbins, c)[0]


@pytest.mark.parametrize("nbins", [2, 5, 100, 4096])
def test_other_grids_follow_their_centres(rule, nbins):
    g = BinGrid.make(1e-3, nbins, 6.0)
    h, c = g.edge_step, np.array(g.centers)
    for e0, eN, step, cc in [
            (g.edge_first, g.edge_last, h, c + 1e-6 * h),
            (g.edge_first, g.edge_last, h, c * 1.01),
            (g.edge_first, g.edge_last - 2 * h, h, c),
            (0.5 * g.edge_first, 0.5 * g.edge_last, 0.5 * h, c)]:
        halves, inv, off = rule(e0, eN, step, cc)
        assert not halves
        # centre k is where cell k + 1 starts
        k = np.arange(nbins)
        assert np.abs(cc * inv + off - (k + 1)).max() <= 1e-12 * nbins
    halves, inv, off = rule(g.edge_last, g.edge_first, -h, c)
    assert not halves
    halves, inv, off = rule(g.edge_first, g.edge_last, h, c[::-1])
    assert not halves and inv == 0.0 and off == nbins


def test_one_centre_off_its_bin_is_flat(rule):
    halves, inv, off = rule(-1.0, 1.0, 2.0, [0.25])
    assert not halves and inv == 0.0 and 0.0 <= off <= 1.0
