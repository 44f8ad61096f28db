"""GPU: setting a state again on a context that keeps its atom count and
settings (list build gated on the device by the type check, one
synchronisation): equal, bit for bit, to a fresh context, in every order of
the calls that follow; a type out of range leaves the state as it was; a
denser state grows the list.  Sizes on both sides of the one-launch build."""
import numpy as np
import pytest

from caviar_b200 import workloads as W

pytestmark = pytest.mark.gpu


def fluid(cells, seed):
    return W.fcc_lattice(cells, 0.8442, 0.9, seed, jitter=0.05)


def ions(n, seed):
    return W.random_ions(n, 16.0, seed, rc=6.0, kmax=4, alpha=0.6)


SYSTEMS = {"lj": lambda seed: fluid(6, seed), "ions": lambda seed: ions(400, seed),
           "large": lambda seed: fluid(26, seed)}  # 70,304 atoms


@pytest.mark.parametrize("kind", list(SYSTEMS))
@pytest.mark.parametrize("prec", [0, 1])
def test_kept_context_equals_a_fresh_one(cuda_lib, kind, prec):
    s, t = SYSTEMS[kind](3), SYSTEMS[kind](4)
    kept, fresh = cuda_lib.Simulation(s, precision=prec), cuda_lib.Simulation(t, precision=prec)
    kept.run(7)
    kept.set_state(t.pos, t.vel, t.type)
    wrong = t.type.copy()
    wrong[-1] = 7
    with pytest.raises(cuda_lib.CvrError):
        kept.set_state(t.pos + 1.0, t.vel, wrong)
    a, th_a = kept.compute_forces()
    b, th_b = fresh.compute_forces()
    assert np.array_equal(a, b) and th_a == th_b
    assert np.array_equal(kept.run(5, 2), fresh.run(5, 2))
    for x, y in zip(kept.state(), fresh.state()):
        assert np.array_equal(x, y)
    # straight into a run, and after a forced build
    kept.set_state(s.pos, s.vel, s.type)
    again = cuda_lib.Simulation(s, precision=prec)
    kept.build_neighbors(True)
    kept.run(4)
    again.run(4)
    for x, y in zip(kept.state(), again.state()):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("prec", [0, 1])
def test_denser_state_grows_the_list(cuda_lib, prec):
    s = W.fcc_lattice(5, 0.3, 0.5, 1)
    sim = cuda_lib.Simulation(s, precision=prec)
    sim.run(2)
    dense = s.pos * 0.75  # in one corner of the box
    sim.set_state(dense, s.vel, s.type)
    acc, _ = sim.compute_forces()
    t = s.copy()
    t.pos = dense
    ref, _ = cuda_lib.Simulation(t, precision=prec).compute_forces()
    assert np.array_equal(acc, ref)
