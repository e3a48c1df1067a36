"""The bounds check of a caller's device array before a kernel may use it in place of a copy
(csrc/hj_ranges.h, covers) on the CPU, at the edges and where sums would wrap, and that
every use of the kernel route asks it with the array's length."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "haissinskijulia_b200", "csrc")
DRIVER = r"""
#include <cstdio>
#include "hj_ranges.h"
int main() {
  unsigned long long a, s, p, n;
  while (scanf("%llu %llu %llu %llu", &a, &s, &p, &n) == 4)
    printf("%d\n", hj_ranges::covers(a, s, p, n) ? 1 : 0);
}
"""
TOP = 2 ** 64


def test_covers(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    (tmp_path / "c.cpp").write_text(DRIVER)
    exe = str(tmp_path / "c")
    subprocess.run([gxx, "-std=c++17", "-I", CSRC, str(tmp_path / "c.cpp"), "-o", exe], check=True)
    cases = [(a, s, p, n)
             for a in (0, 4096, 2 ** 46, TOP - 8192) for s in (0, 8, 4096, 8192)
             for p in (a - 8, a, a + 8, a + s - 8, a + s, a + s + 8, 0, TOP - 8)
             for n in (0, 8, s - 8, s, s + 8, 2 ** 40, TOP - 8) if 0 <= p < TOP and 0 <= n]
    text = "".join("%d %d %d %d\n" % c for c in cases)
    out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout.split()
    assert len(out) == len(cases)
    for (a, s, p, n), got in zip(cases, out):
        assert (got == "1") == (a <= p and p + n <= a + s), (a, s, p, n)


def test_the_kernel_route_asks_for_the_whole_array():
    with open(os.path.join(CSRC, "hj_batch.cu")) as f:
        code = re.sub(r"//[^\n]*", "", f.read())
    calls = re.findall(r"on_device\(ctx, \w+(.*?)\)", code)
    assert len(calls) == 4 and all(c in (", n", ", b->n") for c in calls)
