"""GPU: trajectories whose checkpoints fit the device's free memory without the
forces but not with them: the gradient is the unconstrained one, bit for bit."""
import numpy as np
import pytest

from test_adjoint_memory import MIB, device_memory_left
from test_adjoint_sizes import system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
def test_checkpoints_without_forces(cuda_lib, prec):
    s = system(20000, 2, kmax=1)  # 60 checkpoints of 0.96 MB, 1.44 MB with the forces
    a = cuda_lib.Adjoint.from_system(s, prec)
    J, g = a.loss_grad(120, 2)
    b = cuda_lib.Adjoint.from_system(s, prec)
    b.loss_grad(2, 2)
    with device_memory_left(72 * MIB):
        J1, g1 = b.loss_grad(120, 2)
    assert J == J1
    for k in g:
        assert np.array_equal(g[k], g1[k])
