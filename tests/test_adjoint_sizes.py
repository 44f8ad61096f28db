"""GPU adjoint at the edges of its kernels' splits, against the FP64
restatement (oracle/adjoint.c): atom counts around a warp, a queue and an S(k)
chunk, one species only, no k space, no Ewald term, a real-space cutoff below
the LJ cutoff, and segments that do not divide the trajectory.  Tolerances are
those of tests/test_adjoint.py for the same quantities."""
import dataclasses

import numpy as np
import pytest

from caviar_b200 import workloads as W

pytestmark = pytest.mark.gpu


def system(n, types, kmax=4, rc_r=3.0, k_e=1.0, rc_lj=2.5, seed=1):
    """n atoms on random sites of a cubic grid of spacing 1.1; types: 0, 1 or 2 (mixed)."""
    rng = np.random.default_rng(seed)
    m = max(6, int(np.ceil(n ** (1 / 3))) + 1)
    sites = rng.permutation(m ** 3)[:n]
    pos = 1.1 * (np.stack([sites // (m * m), sites // m % m, sites % m], axis=-1) + 0.5)
    base = W.adjoint_mixture(ncell=2)
    typ = rng.integers(0, 2, n) if types == 2 else np.full(n, types)
    return dataclasses.replace(base, box=1.1 * m, pos=pos + rng.uniform(-0.1, 0.1, pos.shape),
                               vel=rng.normal(size=pos.shape), type=typ.astype(np.int32), rc_lj=rc_lj, rc_r=rc_r,
                               alpha=0.9, kmax=kmax, k_e=k_e)


def close(got, ref, tol):
    scale = max(np.linalg.norm(np.ravel(ref)), 1e-300)
    assert np.linalg.norm(np.ravel(got) - np.ravel(ref)) <= tol * scale, (got, ref)


CASES = [system(2, 2), system(31, 2), system(33, 0), system(64, 1), system(129, 2, kmax=0), system(257, 2, kmax=1),
         system(300, 2, rc_r=1.9), system(300, 2, k_e=0.0), system(577, 2, kmax=10), system(1025, 2, kmax=3)]


@pytest.mark.parametrize("case", range(len(CASES)))
@pytest.mark.parametrize("prec", [1, 0])
def test_forces_and_vjp(cuda_lib, oracle_lib, case, prec):
    s = CASES[case]
    a, o = cuda_lib.Adjoint.from_system(s, prec), oracle_lib.AdjOracle(s)
    f, e, dU = a.forces()
    f0, e0, dU0 = o.forces(s.pos)
    u = np.random.default_rng(3).normal(size=s.pos.shape)
    w, g = a.force_vjp(u)
    w0, g0 = o.force_vjp(s.pos, u)
    tol = 1e-10 if prec else 1e-5
    close(f, f0, tol)
    close(w, w0, tol)
    assert np.all(np.abs(e - e0) <= tol * np.maximum(1.0, np.abs(e0)))
    for k in ("eps", "sigma", "charge"):
        close(dU[k], dU0[k], tol)
        # the VJP's parameter gradients are sums of terms of either sign, whose
        # FP32 rounding is relative to the terms: compared in FP64 only
        if prec:
            close(g[k], g0[k], tol)


@pytest.mark.parametrize("prec", [1, 0])
@pytest.mark.parametrize("steps,every", [(1, 1), (5, 5), (7, 3), (6, 10)])
def test_segments(cuda_lib, oracle_lib, prec, steps, every):
    s = CASES[6]
    J0, g0 = oracle_lib.AdjOracle(s).loss_grad(s.pos, s.vel, steps, every)
    J, g = cuda_lib.Adjoint.from_system(s, prec).loss_grad(steps, every)
    tol = 1e-9 if prec else 1e-4
    assert abs(J - J0) <= tol * abs(J0)
    for k in ("pos", "vel", "eps", "sigma", "charge"):
        close(g[k], g0[k], tol)


@pytest.mark.parametrize("prec", [1, 0])
def test_position_that_is_not_finite(cuda_lib, prec):
    s = dataclasses.replace(CASES[4], pos=CASES[4].pos.copy())
    s.pos[7, 1] = np.nan
    f, _, _ = cuda_lib.Adjoint.from_system(s, prec).forces()
    assert np.isnan(f).any(axis=1).all()
