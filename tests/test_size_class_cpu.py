"""Sizes of the context's cached blocks (csrc/hj_ranges.h) on the CPU: a quarter of a power
of two apart up to what the cache keeps, the request's own pages beyond it."""
import os
import random
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "haissinskijulia_b200", "csrc")
DRIVER = r"""
#include <cstdio>
#include "hj_ranges.h"
int main() {
  unsigned long long b, kept;
  while (scanf("%llu %llu", &b, &kept) == 2)
    printf("%llu\n", (unsigned long long)hj_ranges::size_class(b, kept));
}
"""


@pytest.mark.parametrize("kept", [256 << 20, 8 << 30])
def test_size_class(tmp_path, kept):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    (tmp_path / "s.cpp").write_text(DRIVER)
    exe = str(tmp_path / "s")
    subprocess.run([gxx, "-std=c++17", "-I", CSRC, str(tmp_path / "s.cpp"), "-o", exe], check=True)
    rng = random.Random(kept)
    sizes = [0, 1, 4095, 4096, 4097, kept - 1, kept, kept + 1, 150 << 30, (160 << 30) + 1]
    sizes += [int(2 ** rng.uniform(0, 38)) for _ in range(2000)]
    out = subprocess.run([exe], input="".join(f"{b} {kept}\n" for b in sizes),
                         capture_output=True, text=True, check=True).stdout.split()
    for b, c in zip(sizes, map(int, out)):
        assert c >= max(b, 4096) and c % 1024 == 0
        if b <= 4096:
            assert c == 4096
        elif b <= kept:
            assert c <= 1.25 * b and c * 8 % (1 << (c.bit_length() - 1)) == 0
        else:
            assert c - b < 4096
