"""GPU: the replica batch's state in and out (reordered on the device, charged
atoms first): every atom comes back to its place bit for bit, for replicas
around the sizes of a block round, all neutral, all charged and mixed; a type
out of range is refused and leaves the state as it was."""
import numpy as np
import pytest

from caviar_b200 import workloads as W

pytestmark = pytest.mark.gpu
SIZES = [1, 2, 31, 255, 256, 257, 511, 513, 2048]


@pytest.mark.parametrize("charges", ["none", "all", "mixed"])
def test_round_trip(cuda_lib, charges):
    b = W.replica_batch(sizes=SIZES, seed=9)
    rng = np.random.default_rng(1)
    n = len(b.type)
    typ = {"none": np.zeros(n), "all": 1 + np.arange(n) % 2, "mixed": rng.integers(0, 3, n)}[charges].astype(np.int32)
    h = cuda_lib.Batch(b.n, b.box, np.array([1.0, 2.0, 4.0]), b.charge)
    h.set_forces(b.epsilon, b.sigma, b.rc_lj, b.rc_r, b.alpha, b.kmax, b.k_e, b.dt)
    h.set_state(b.pos, b.vel, typ)
    pos, vel, _ = h.state()
    assert np.array_equal(pos, b.pos) and np.array_equal(vel, b.vel)
    wrong = typ.copy()
    wrong[-1] = 3
    with pytest.raises(cuda_lib.CvrError):
        h.set_state(b.pos + 1.0, b.vel, wrong)
    pos, vel, _ = h.state()
    assert np.array_equal(pos, b.pos) and np.array_equal(vel, b.vel)
    # one run from a new state equals a zero-step run and a run
    h.run(5)
    one = h.state()
    h.set_state(b.pos, b.vel, typ)
    h.run(0)
    h.run(5)
    for x, y in zip(one, h.state()):
        assert np.array_equal(x, y)
