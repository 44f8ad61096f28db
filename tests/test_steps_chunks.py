"""GPU: long runs of small systems go in several launches, so that other streams
are not kept waiting for seconds, with the bits of one kernel per stage across
their ends; and two contexts that run at the same time, one thread each, get
what they get alone."""
import threading

import numpy as np
import pytest

from test_steps_in_one_launch import both, system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,steps,launches", [(33, 2500, 3), (20001, 1700, 3)])
def test_launches_of_a_long_run(cuda_lib, n, steps, launches):
    sim = cuda_lib.Simulation(system(n))
    sim.run(1)
    before = sim.launches
    sim.run(steps)
    assert launches <= sim.launches - before <= launches + 4


@pytest.mark.parametrize("kind", ["lj", "mixture"])
@pytest.mark.parametrize("every", [0, 7])
def test_equal_across_launches(cuda_lib, kind, every):
    a, b = both(cuda_lib, system(150, kind), 0, [2100], every)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


def test_two_contexts_at_once(cuda_lib):
    systems = [system(3000, seed=1), system(20001, seed=2)]

    def run(s, out, k):
        sim = cuda_lib.Simulation(s)
        for _ in range(8):
            sim.set_state(s.pos, s.vel, s.type)
            sim.run(150)
        out[k] = sim.state()

    alone, together = {}, {}
    for k, s in enumerate(systems):
        run(s, alone, k)
    threads = [threading.Thread(target=run, args=(s, together, k)) for k, s in enumerate(systems)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(2):
        for x, y in zip(alone[k], together[k]):
            assert np.array_equal(x, y)
