"""The batch's rule for particles per block (csrc/hj_launch.h, member_chunk) on
the CPU: blocks cover the bunch, start on whole warps of four-particle groups (so
that the 32-byte loads stay aligned), stay within twice the batch's chunk and the
per-block bound, and no bunch takes more blocks than the batch's tables hold."""
import os
import random
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "haissinskijulia_b200", "csrc")
DRIVER = r"""
#include <cstdio>
#include "hj_launch.h"
int main() {
  long long n, chunk, slots;
  printf("%lld\n", (long long)hj::kMaxBlockParticles);
  while (scanf("%lld %lld %lld", &n, &chunk, &slots) == 3)
    printf("%lld %lld\n", (long long)hj::member_chunk(n, chunk, slots),
           (long long)hj::member_blocks(slots));
}
"""


@pytest.mark.parametrize("chunk", [4, 100, 4096, 16384, 65536, 65540, 262144, 2**20 - 8])
def test_member_chunk(tmp_path, chunk):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    (tmp_path / "m.cpp").write_text(DRIVER)
    exe = str(tmp_path / "m")
    subprocess.run([gxx, "-std=c++17", "-I", CSRC, str(tmp_path / "m.cpp"), "-o", exe], check=True)
    rng = random.Random(chunk)
    ns = [1, 2, 127, 128, 129, 16383, 16384, 16385, 131071, 131072, 131073, 2**20, 10**8]
    ns += [rng.randrange(1, 2**24) for _ in range(200)]
    cases = [(n, slots) for n in ns for slots in (1, 2, 16, 37, 148, 1000)]
    out = subprocess.run([exe], input="".join(f"{n} {chunk} {s}\n" for n, s in cases),
                         capture_output=True, text=True, check=True).stdout.split()
    most = int(out[0])
    for (n, slots), c, blocks in zip(cases, map(int, out[1::2]), map(int, out[2::2])):
        assert 0 < c <= min(2 * chunk, most)
        assert c % 4 == 0
        assert -(-n // c) <= n // chunk + blocks + 1, (n, c)
