"""A batch's blocks of particles (csrc/hj_launch.h, member_chunk to member_end) on the CPU:
a caller's own chunk is the block size, the default leaves it to the library's rule; the
blocks cover the bunch and start on whole warps, and the sizes the autotuner tries split a
workload differently."""
import os
import shutil
import subprocess

import pytest

from haissinskijulia_b200.sweep import intensity_scan, sweep_points, wave_chunks

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "haissinskijulia_b200", "csrc")
DRIVER = r"""
#include <cstdio>
#include "hj_launch.h"
int main() {
  long long n, chunk, slots;
  long long sms;
  while (scanf("%lld %lld %lld %lld", &n, &chunk, &slots, &sms) == 4) {
    const int64_t c = hj::member_chunk(n, chunk, slots, sms), k = hj::member_chunks(n, c);
    printf("%lld %lld", (long long)c, (long long)k);
    for (int64_t i = 0; i < k; ++i)
      printf(" %lld %lld", (long long)hj::member_first(i, c), (long long)hj::member_end(i, n, c));
    printf("\n");
  }
}
"""


@pytest.fixture(scope="module")
def split(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("split")
    (d / "s.cpp").write_text(DRIVER)
    exe = str(d / "s")
    subprocess.run([gxx, "-std=c++17", "-I", CSRC, str(d / "s.cpp"), "-o", exe], check=True)

    def run(cases, sms=148):
        text = "".join("%d %d %d %d\n" % (*c, sms) for c in cases)
        out = subprocess.run([exe], input=text,
                             capture_output=True, text=True, check=True).stdout.splitlines()
        rows = []
        for line in out:
            v = [int(x) for x in line.split()]
            rows.append((v[0], list(zip(v[2::2], v[3::2]))))
            assert len(rows[-1][1]) == v[1]
        return rows
    return run


SIZES = [1, 3, 127, 128, 129, 16383, 16384, 54056, 54057, 65536, 108112, 131073, 600_000, 999_983,
         2_000_000, 7 * 2**20]


@pytest.mark.parametrize("chunk", [4, 100, 128, 4096, 16384, 54056, 65536, 108112, 262144, 2**20 - 128,
                                   2**20 - 64, 2**20 - 8])
def test_blocks_cover_the_bunch_on_whole_warps(split, chunk):
    cases = [(n, chunk, s) for n in SIZES for s in (1, 16, 256)]
    for (n, _, _), (c, blocks) in zip(cases, split(cases)):
        assert blocks[0][0] == 0 and blocks[-1][1] == n
        assert all(a[1] == b[0] for a, b in zip(blocks, blocks[1:]))
        for first, end in blocks:
            assert first % (128 if c >= 128 else 4) == 0
            assert 0 < end - first <= 2**20 - 8
        if chunk != 65536:
            assert c == (chunk if chunk < 2**20 - 256 else 2**20 - 128)
            assert all(abs(e - f - c) < 128 for f, e in blocks[:-1])


def test_the_default_does_not_depend_on_other_bunches_and_fills_the_gpu(split):
    for n, slots, want in [(10_000, 256, 1), (1_000_000, 32, 9), (2_000_000, 256, 16),
                           (1_600_000, 16, 18)]:
        assert len(split([(n, 65536, slots)])[0][1]) == want


@pytest.mark.parametrize("points", [intensity_scan(), sweep_points(64)])
def test_the_autotuner_tries_different_splits(split, points):
    chunks = sorted(set([16384, 65536, 262144] + wave_chunks(points, 148)))
    seen = {tuple(len(b) for _, b in split([(p.n, c, len(points)) for p in points]))
            for c in chunks}
    assert len(seen) == len(chunks)


def test_the_default_follows_the_number_of_sms(split):
    for sms in (37, 74, 148):
        assert len(split([(10_000_000, 65536, 2)], sms)[0][1]) == max(sms, -(-10_000_000 // 131072))
        assert len(split([(1_000_000, 65536, 32)], sms)[0][1]) == max(8, 2 * sms // 32)
