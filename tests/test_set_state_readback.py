"""GPU: what is read back right after a state is set again on a kept context
(accelerations, S(k)) belongs to that state: equal, bit for bit, to what a
fresh context computes from it, and the run that follows is the same with and
without the reading."""
import numpy as np
import pytest

from test_set_state import SYSTEMS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", list(SYSTEMS))
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("first", ["acc", "sk"])
def test_readback_after_set_state(cuda_lib, kind, prec, first):
    s, t = SYSTEMS[kind](3), SYSTEMS[kind](4)
    kept, fresh = cuda_lib.Simulation(s, precision=prec), cuda_lib.Simulation(t, precision=prec)
    kept.run(3)
    kept.set_state(t.pos, t.vel, t.type)
    acc, _ = fresh.compute_forces()
    if first == "sk":
        assert np.array_equal(kept.sk(), fresh.sk())
    assert np.array_equal(kept.state()[2], fresh.state()[2])
    assert np.array_equal(kept.sk(), fresh.sk())
    # compute_forces returns accelerations in the caller's order, as state() does
    assert np.array_equal(kept.state()[2], acc)
    assert np.array_equal(kept.run(5, 2), fresh.run(5, 2))
    for x, y in zip(kept.state(), fresh.state()):
        assert np.array_equal(x, y)
