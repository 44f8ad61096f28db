"""GPU: settings refused after the context began to follow them (a neighbour
cutoff that gives too many cells) are refused again by every call that would use
them, and acceptable settings make the context work as a fresh one."""
import numpy as np
import pytest

from test_set_state import SYSTEMS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["lj", "ions"])
@pytest.mark.parametrize("prec", [0, 1])
def test_too_many_cells(cuda_lib, kind, prec):
    def code(call):
        with pytest.raises(cuda_lib.CvrError) as e:
            call()
        return e.value.code

    s = SYSTEMS[kind](3)
    sim, fresh = (cuda_lib.Simulation(s, precision=prec) for _ in range(2))
    tiny = s.box.min() / 1000.0
    assert code(lambda: sim._check(sim.L.cvr_set_neighborlist(sim.h, tiny, 1.0, tiny, 0))) == 5
    for call in (lambda: sim.run(1), sim.compute_forces, sim.build_neighbors):
        assert code(call) == 5
    assert code(sim.pairs) == 4
    sim._check(sim.L.cvr_set_neighborlist(sim.h, s.cutoff, s.coef, s.ghost_cutoff, 0))
    assert np.array_equal(sim.run(5, 2), fresh.run(5, 2))
    for x, y in zip(sim.state(), fresh.state()):
        assert np.array_equal(x, y)
