"""GPU: a state set before its Ewald terms is computed as one set after them
(the same lanes per atom, the same bits), and again after the terms changed."""
import dataclasses

import numpy as np
import pytest

from caviar_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n", [4144, 4145, 9000])
def test_ewald_after_the_state(cuda_lib, n, prec):
    s = W.random_ions(n, 26.0 * (n / 8000.0) ** (1.0 / 3.0), 2, rc=5.0, kmax=3, alpha=0.7)
    late = cuda_lib.Simulation(dataclasses.replace(s, ewald_r=None, ewald_k=None), precision=prec)
    late.run(0)
    late.configure(s, cuda_lib.REBUILD_DISPLACEMENT)
    ref = cuda_lib.Simulation(s, precision=prec)
    assert late.info()["tpa"] == ref.info()["tpa"] == 32
    a, b = late.run(12, 4), ref.run(12, 4)
    a[:, -1] -= 1  # the list builds: one for the system without the terms
    assert np.array_equal(a, b)
    for x, y in zip(late.state(), ref.state()):
        assert np.array_equal(x, y)
    late.set_state(s.pos, s.vel, s.type)
    assert np.array_equal(late.compute_forces()[0], cuda_lib.Simulation(s, precision=prec).compute_forces()[0])
