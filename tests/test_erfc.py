"""GPU: the FP64 Ewald real-space energy and force of one ion pair against
mpmath over the range of alpha r that cutoffs reach.  Tolerance: the polynomial
is within 6.5e-16 relative, each of the about ten roundings of exp, reciprocal
and products adds 1.2e-16, and exp(-x^2) has the rounding of its argument,
2 x^2 1.2e-16: below (3e-15 + 3e-16 x^2) relative."""
import dataclasses

import mpmath
import numpy as np
import pytest

from caviar_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alpha", [0.02, 0.3, 1.1, 3.0])
@pytest.mark.parametrize("r", [0.03, 0.4, 1.0, 2.7, 4.9])
def test_pair(cuda_lib, alpha, r):
    base = W.adjoint_mixture(ncell=2)
    s = dataclasses.replace(base, box=10.0, pos=np.array([[1.0, 1.0, 1.0], [1.0 + r, 1.0, 1.0]]), vel=np.zeros((2, 3)),
                            type=np.array([0, 1], np.int32), epsilon=np.zeros((2, 2)), alpha=alpha, rc_r=5.0, kmax=0)
    f, e, _ = cuda_lib.Adjoint.from_system(s, 1).forces()
    d = mpmath.mpf(float(s.pos[1, 0])) - mpmath.mpf(1)
    x = mpmath.mpf(alpha) * d
    qq = mpmath.mpf(float(s.charge[0] * s.charge[1]))
    energy = qq * mpmath.erfc(x) / d
    force = qq * (2 * mpmath.mpf(alpha) / mpmath.sqrt(mpmath.pi) * mpmath.exp(-x * x) + mpmath.erfc(x) / d) / d
    tol = 3e-15 + 3e-16 * float(x * x)
    assert abs(e[1] - float(energy)) <= tol * abs(float(energy))
    assert abs(f[1, 0] - float(force)) <= tol * abs(float(force))
    assert f[0, 0] == -f[1, 0]
