"""GPU: launches whose blocks wait for one another (many steps, a list build)
that fail or are refused, on the host's request.  A failed launch leaves the
state and the barrier words as they were: the call made again gives what an
undisturbed context gives, bit for bit.  A refused one is replaced by one kernel
per stage, with the same results."""
import numpy as np
import pytest

from test_set_state import SYSTEMS
from test_steps_in_one_launch import system

pytestmark = pytest.mark.gpu

TOO_LARGE, NOT_SUPPORTED, UNKNOWN = 720, 801, 999  # cudaError_t


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n", [3, 500, 6001])
def test_failed_launch_of_a_run(cuda_lib, n, prec):
    s = system(n)
    sim, fresh = (cuda_lib.Simulation(s, precision=prec) for _ in range(2))
    for steps in (4, 1, 7, 3):
        sim.inject_failure(cuda_lib.INJECT_LAUNCH_ERROR, UNKNOWN)
        with pytest.raises(cuda_lib.CvrError) as e:
            sim.run(steps, 2)
        assert e.value.code == 2
        assert np.array_equal(sim.run(steps, 2), fresh.run(steps, 2))
        for x, y in zip(sim.state(), fresh.state()):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("code", [TOO_LARGE, NOT_SUPPORTED])
@pytest.mark.parametrize("n", [500, 6001])
def test_refused_launch_of_a_run(cuda_lib, n, code, prec):
    s = system(n)
    sim, fresh = (cuda_lib.Simulation(s, precision=prec) for _ in range(2))
    assert np.array_equal(sim.run(5, 2), fresh.run(5, 2))
    sim.inject_failure(cuda_lib.INJECT_LAUNCH_ERROR, code)
    for steps in (20, 5):
        before = sim.launches
        assert np.array_equal(sim.run(steps, 3), fresh.run(steps, 3))
        assert sim.launches - before > steps  # one kernel per stage
        for x, y in zip(sim.state(), fresh.state()):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("kind", ["lj", "ions"])
@pytest.mark.parametrize("prec", [0, 1])
def test_refused_launch_of_a_build(cuda_lib, kind, prec):
    s, t = SYSTEMS[kind](3), SYSTEMS[kind](4)
    sim, fresh = cuda_lib.Simulation(s, precision=prec), cuda_lib.Simulation(t, precision=prec)
    sim.run(2)
    sim.inject_failure(cuda_lib.INJECT_LAUNCH_ERROR, TOO_LARGE)
    sim.set_state(t.pos, t.vel, t.type)
    assert np.array_equal(sim.compute_forces()[0], fresh.compute_forces()[0])
    assert np.array_equal(sim.run(5, 2), fresh.run(5, 2))
    for x, y in zip(sim.state(), fresh.state()):
        assert np.array_equal(x, y)
