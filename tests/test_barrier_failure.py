"""GPU: a wait between the blocks of a many-step launch, or of a list build,
that runs out (one poll allowed, on the host's request) fails the call and
leaves a context that refuses to go on with the half-done state, takes a new
one, and then computes what a fresh context computes, bit for bit."""
import numpy as np
import pytest

from test_set_state import SYSTEMS

pytestmark = pytest.mark.gpu


def failed(abi, call):
    with pytest.raises(abi.CvrError) as e:
        call()
    return e.value.code


def check(abi, sim, s, prec):
    sim.inject_failure(abi.INJECT_BARRIER_POLLS, 0)
    assert failed(abi, lambda: sim.run(1)) == 4  # no state
    assert failed(abi, sim.state) == 4
    assert failed(abi, sim.compute_forces) == 4
    sim.set_state(s.pos, s.vel, s.type)
    fresh = abi.Simulation(s, precision=prec)
    for _ in range(2):
        assert np.array_equal(sim.run(6, 3), fresh.run(6, 3))
        for x, y in zip(sim.state(), fresh.state()):
            assert np.array_equal(x, y)
    # and again on the kept context
    sim.set_state(s.pos, s.vel, s.type)
    again = abi.Simulation(s, precision=prec)
    assert np.array_equal(sim.compute_forces()[0], again.compute_forces()[0])


@pytest.mark.parametrize("prec", [0, 1])
def test_run(cuda_lib, prec):
    s, t = SYSTEMS["lj"](3), SYSTEMS["lj"](4)
    sim = cuda_lib.Simulation(s, precision=prec)
    sim.run(5)
    sim.inject_failure(cuda_lib.INJECT_BARRIER_POLLS, 1)
    assert failed(cuda_lib, lambda: sim.run(20)) == 2
    check(cuda_lib, sim, t, prec)


@pytest.mark.parametrize("kind", ["lj", "ions"])
@pytest.mark.parametrize("prec", [0, 1])
def test_set_state(cuda_lib, kind, prec):
    s, t = SYSTEMS[kind](3), SYSTEMS[kind](4)
    sim = cuda_lib.Simulation(s, precision=prec)
    sim.run(2)
    sim.inject_failure(cuda_lib.INJECT_BARRIER_POLLS, 1)
    assert failed(cuda_lib, lambda: sim.set_state(t.pos, t.vel, t.type)) == 2
    check(cuda_lib, sim, t, prec)


def test_precision_after_a_failure(cuda_lib):
    s = SYSTEMS["lj"](3)
    sim = cuda_lib.Simulation(s, precision=0)
    sim.inject_failure(cuda_lib.INJECT_BARRIER_POLLS, 1)
    assert failed(cuda_lib, lambda: sim.run(20)) == 2
    sim.inject_failure(cuda_lib.INJECT_BARRIER_POLLS, 0)
    cuda_lib.load().cvr_set_precision(sim.h, 1)
    sim.set_state(s.pos, s.vel, s.type)
    fresh = cuda_lib.Simulation(s, precision=1)
    sim.run(4), fresh.run(4)
    for x, y in zip(sim.state(), fresh.state()):
        assert np.array_equal(x, y)
