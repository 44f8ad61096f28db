"""GPU: a cvr_set_state with another atom count that is refused (a type out of
range) has given up the old state's arrays: every call that needs a state says
so, and the next state is computed as on a fresh context."""
import numpy as np
import pytest

from test_set_state import ions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n", [300, 700])
def test_refused_state_of_another_size(cuda_lib, n, prec):
    def code(call):
        with pytest.raises(cuda_lib.CvrError) as e:
            call()
        return e.value.code

    s, t = ions(400, 3), ions(n, 4)
    wrong = t.type.copy()
    wrong[0] = -1
    sim = cuda_lib.Simulation(s, precision=prec)
    sim.run(2)
    assert code(lambda: sim.set_state(t.pos, t.vel, wrong)) == 1
    for call in (lambda: sim.run(1), sim.compute_forces, sim.state, sim.build_neighbors, sim.pairs):
        assert code(call) == 4
    sim.set_state(t.pos, t.vel, t.type)
    fresh = cuda_lib.Simulation(t, precision=prec)
    assert np.array_equal(sim.run(5, 2), fresh.run(5, 2))
    for x, y in zip(sim.state(), fresh.state()):
        assert np.array_equal(x, y)
