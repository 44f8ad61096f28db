"""GPU: a cvr_set_state that fails after the new positions were written (its
list build cannot be launched, on the host's request) leaves no state: every
call that needs one says so, until a state is set; a type out of range still
leaves the state as it was."""
import numpy as np
import pytest

from test_set_state import SYSTEMS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["lj", "ions"])
@pytest.mark.parametrize("prec", [0, 1])
def test_failed_set_state(cuda_lib, kind, prec):
    def code(call):
        with pytest.raises(cuda_lib.CvrError) as e:
            call()
        return e.value.code

    s, t = SYSTEMS[kind](3), SYSTEMS[kind](4)
    wrong = t.type.copy()
    wrong[-1] = 7
    sim, fresh = cuda_lib.Simulation(s, precision=prec), cuda_lib.Simulation(t, precision=prec)
    sim.run(3)
    before, pairs = sim.state(), sim.pairs()
    assert code(lambda: sim.set_state(t.pos, t.vel, wrong)) == 1
    for x, y in zip(before, sim.state()):
        assert np.array_equal(x, y)
    assert np.array_equal(pairs, sim.pairs())
    sim.inject_failure(cuda_lib.INJECT_LAUNCH_ERROR, 999)
    assert code(lambda: sim.set_state(t.pos, t.vel, t.type)) == 2
    for call in (lambda: sim.run(1), sim.compute_forces, sim.state, sim.build_neighbors, sim.pairs):
        assert code(call) == 4
    assert code(lambda: sim.set_state(t.pos, t.vel, wrong)) == 1
    assert code(lambda: sim.run(1)) == 4
    sim.set_state(t.pos, t.vel, t.type)
    assert np.array_equal(sim.run(5, 2), fresh.run(5, 2))
    for x, y in zip(sim.state(), fresh.state()):
        assert np.array_equal(x, y)
