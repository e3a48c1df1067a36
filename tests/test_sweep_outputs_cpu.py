"""The host arrays of run_batched(copy_out=True) on the CPU: each point's are its own, and
the thread that has their pages mapped leaves alone what was handed out."""
import gc
import weakref

import numpy as np

from haissinskijulia_b200 import sweep
from haissinskijulia_b200.sweep import Point


def _points(ns):
    return [Point(n, 5e6, 1e10, 64, 1, i) for i, n in enumerate(ns)]


def test_every_solve_owns_its_particles():
    out = sweep._Outputs(_points([1, 7, 513, 100_000, 0]))
    pairs = [out.of(i) for i in range(5)]
    for (z, dE), n in zip(pairs, [1, 7, 513, 100_000, 0]):
        assert z.shape == dE.shape == (n,) and z.dtype == dE.dtype == np.float64
        assert z.base is None and dE.base is None
    out._thread.join()
    kept = pairs[1]
    refs = [weakref.ref(a) for i in (0, 2, 3) for a in pairs[i]]
    del pairs, out, z, dE
    gc.collect()
    assert all(r() is None for r in refs)
    assert kept[0].shape == (7,)


def test_results_are_not_touched():
    n = 3_000_000
    for _ in range(3):
        out = sweep._Outputs(_points([n] * 6))
        taken = []
        for i in (5, 0, 3, 1):
            z, dE = out.of(i)
            z[:] = i + 1.0
            dE[:] = -i - 1.0
            taken.append((i, z, dE))
        out._thread.join()
        for i, z, dE in taken:
            assert (z == i + 1.0).all() and (dE == -i - 1.0).all()
