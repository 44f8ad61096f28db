"""GPU: the mixed adjoint's accuracy does not depend on the box: one cluster of
300 atoms at random places of boxes from 11 to 10^5 LJ diameters (fixed-point
and FP64 pair differences, and both sides of the line between them), against
the FP64 restatement (oracle/adjoint.c).

Tolerance: a displacement is rounded once to FP32 (2^-24 relative at most),
which the r^-13 force at contact amplifies 14 times, 8.4e-7, and about ten
FP32 operations add 1e-7 (r.m.s.): 1e-6 of the norm.  A position that is not
finite makes every force NaN in both forms."""
import dataclasses

import numpy as np
import pytest

from test_adjoint_sizes import system

pytestmark = pytest.mark.gpu


def cluster(box, seed):
    s = system(300, 2, kmax=2, seed=seed)
    off = np.random.default_rng(seed).uniform(0, box, 3)
    return dataclasses.replace(s, box=box, pos=s.pos + off)


@pytest.mark.parametrize("box", [11.0, 24.0, 31.0, 33.0, 100.0, 1e3, 1e5])
@pytest.mark.parametrize("seed", [1, 2])
def test_cluster(cuda_lib, oracle_lib, box, seed):
    s = cluster(box, seed)
    a, o = cuda_lib.Adjoint.from_system(s, 0), oracle_lib.AdjOracle(s)
    f, e, _ = a.forces()
    f0, e0, _ = o.forces(s.pos)
    u = np.random.default_rng(3).normal(size=s.pos.shape)
    w, w0 = a.force_vjp(u)[0], o.force_vjp(s.pos, u)[0]
    assert np.linalg.norm(f - f0) <= 1e-6 * np.linalg.norm(f0)
    assert np.linalg.norm(w - w0) <= 1e-6 * np.linalg.norm(w0)
    assert abs(e[0] - e0[0]) <= 1e-6 * abs(e0[0])


@pytest.mark.parametrize("box", [11.0, 1e3])
def test_position_that_is_not_finite(cuda_lib, box):
    s = cluster(box, 1)
    s.pos[7, 1] = np.nan
    f, e, _ = cuda_lib.Adjoint.from_system(s, 0).forces()
    assert np.isnan(f).any(axis=1).all()
    assert np.isnan(e[1])
