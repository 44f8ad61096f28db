"""GPU: thermostats at atom counts whose blocks hold one to three warps (fewer
than the four sums of a thermostat) in the launch that runs many steps, against
the one-kernel-per-stage path, FP64.  The kinetic energy is summed in another
order: 1e-14 per step, times 25 steps, times the growth of a perturbation over
0.125 time units (below 10), within 1e-10 of the velocities."""
import numpy as np
import pytest

from test_steps_in_one_launch import both, system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["berendsen", "nose_hoover"])
@pytest.mark.parametrize("n", [2, 3, 5, 6, 9, 13])
def test_thermostats(cuda_lib, kind, n):
    def setup(sim):
        if kind == "berendsen":
            sim.set_berendsen(1.2, 0.1, 0.005, step=2)
        else:
            sim.set_nose_hoover(1.2, 0.005, type=1, mass=20.0, kb=1.0)
    a, b = both(cuda_lib, system(n, "mixture"), 1, [10, 15], 5, setup=setup)
    assert np.abs(a[1] - b[1]).max() <= 1e-10
    assert np.allclose(a[3], b[3], rtol=1e-9, atol=1e-9)
    assert a[4] == b[4]
