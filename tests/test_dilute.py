"""GPU: systems with many more cells than atoms, on both sides of the line (128
cells per thread) up to which a list is built inside one launch: lists equal to
the oracle's, and runs with rebuilds equal, bit for bit, to one kernel per
stage; at no density does the build cost what a sum over all cells per block
would (less than three times the staged build's time)."""
import time

import numpy as np
import pytest

from caviar_b200 import workloads as W
from test_steps_in_one_launch import both, system

pytestmark = pytest.mark.gpu


def gas(n, cells):
    """n atoms of a hot gas in a box of cells^3 list cells (1.4 wide: half of cutoff and skin)."""
    s = system(n)
    length = 1.4 * cells + 0.5
    s.pos, s.vel = s.pos * (length / s.hi), 4.0 * s.vel
    s.hi = np.full(3, length)
    return s


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n,cells", [(2, 19), (2, 21), (9, 40), (100, 50), (100, 74), (100, 75), (500, 60), (4145, 90)])
def test_runs(cuda_lib, n, cells, prec):
    a, b = both(cuda_lib, gas(n, cells), prec, [1, 24], 8)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
    assert a[4] > 3


@pytest.mark.parametrize("n,cells", [(9, 40), (500, 60), (4000, 50)])
def test_pairs(cuda_lib, oracle_lib, n, cells):
    s = gas(n, cells)
    s.pos[1::2] = s.pos[::2][: n // 2] + np.array([1.0, 0.2, 0.1])  # pairs in contact
    o = oracle_lib.Oracle(s)
    o.setup()
    sim = cuda_lib.Simulation(s)
    sim.build_neighbors(True)
    assert np.array_equal(sim.pairs(), o.pairs())


@pytest.mark.parametrize("n,cells", [(100, 75), (500, 60), (500, 120), (4000, 110)])
def test_build_time(cuda_lib, n, cells):
    sim = cuda_lib.Simulation(gas(n, cells))

    def build():
        t = []
        for _ in range(20):
            t0 = time.perf_counter()
            sim.build_neighbors(True)
            t.append(time.perf_counter() - t0)
        return np.median(t)

    build()
    one = build()
    sim.inject_failure(cuda_lib.INJECT_LAUNCH_ERROR, 720)  # one kernel per stage from here on
    build()
    assert one < 3.0 * build()
