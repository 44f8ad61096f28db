"""GPU: replicas on both sides of the lines that decide whether a replica has an
LJ list (atoms, expected partners within the cutoff and the skin, the charged
share), forces and energies against the FP64 replica oracle with the tolerances
of tests/test_batch.py; cutoffs changed on one handle; a batch whose lists do
not fit the device's free memory runs with all pairs; and no replica takes
longer than with all pairs."""
import time

import numpy as np
import pytest

from caviar_b200 import workloads as W
from helpers import force_errors
from test_adjoint_memory import MIB, device_memory_left
from test_batch import ENERGY_TOL, FORCE_TOL, MAX_TOL, make_batch, oracle_forces, replica

pytestmark = pytest.mark.gpu


def batch(sizes, charged, cutoff):
    b = W.replica_batch(sizes=sizes, seed=9, lj_cutoff=cutoff)
    rng = np.random.default_rng(3)
    b.type = np.concatenate([np.where(np.arange(n) < round(charged * n), 1 + np.arange(n) % 2, 0)[rng.permutation(n)]
                             for n in sizes]).astype(np.int32)
    return b


def check(O, b, h):
    out = h.run(0)
    acc = h.state()[2]
    for r in range(len(b.n)):
        ref, en = oracle_forces(O, b, r)
        g, m, _ = force_errors(acc[replica(b, r)], ref)
        assert g < FORCE_TOL and m < MAX_TOL, (b.n[r], g, m)
        got = dict(zip(h.OUT_KEYS, out[r]))
        for k in ("e_lj", "e_ewald_r", "virial"):
            assert abs(got[k] - en[k]) <= ENERGY_TOL * max(1.0, abs(en[k])), (b.n[r], k)


@pytest.mark.parametrize("charged", [0.0, 0.69, 0.71, 1.0])
@pytest.mark.parametrize("cutoff", [1.2, 2.5, 2.85, 2.9, 3.2])
def test_forces_and_energies(cuda_lib, oracle_lib, charged, cutoff):
    b = batch([191, 192, 400], charged, cutoff)
    check(oracle_lib, b, make_batch(cuda_lib, b))


def test_cutoffs_changed_on_one_handle(cuda_lib, oracle_lib):
    b = batch([150, 300, 500], 0.5, 3.2)
    h = make_batch(cuda_lib, b)
    for cutoff in (3.2, 1.5, 2.5, 3.2, 2.8):
        b.rc_lj = np.minimum(cutoff, b.box / 2)
        h.set_forces(b.epsilon, b.sigma, b.rc_lj, b.rc_r, b.alpha, b.kmax, b.k_e, b.dt)
        check(oracle_lib, b, h)


def test_lists_that_do_not_fit(cuda_lib, oracle_lib):
    b = batch([300] * 400, 0.5, 2.5)  # 32.6 MB of lists
    h = cuda_lib.Batch(b.n, b.box, b.mass, b.charge)
    with device_memory_left(16 * MIB):
        h.set_forces(b.epsilon, b.sigma, b.rc_lj, b.rc_r, b.alpha, b.kmax, b.k_e, b.dt)
    h.set_state(b.pos, b.vel, b.type)
    out = h.run(0)
    few = make_batch(cuda_lib, b)
    assert np.allclose(out, few.run(0), rtol=1e-5, atol=1e-3)


@pytest.mark.parametrize("charged,cutoff", [(1.0, 2.5), (0.5, 3.0), (0.0, 3.5), (0.5, 2.5)])
def test_no_slower_than_all_pairs(cuda_lib, charged, cutoff):
    b = batch([600] * 148, charged, cutoff)
    free = cuda_lib.Batch(b.n, b.box, b.mass, b.charge)
    free.set_forces(b.epsilon, b.sigma, b.rc_lj, b.rc_r, b.alpha, b.kmax, b.k_e, b.dt)
    tiles = cuda_lib.Batch(b.n, b.box, b.mass, b.charge)
    with device_memory_left(4 * MIB):  # no room for lists
        tiles.set_forces(b.epsilon, b.sigma, b.rc_lj, b.rc_r, b.alpha, b.kmax, b.k_e, b.dt)
    t = []
    for h in (free, tiles):
        h.set_state(b.pos, b.vel, b.type)
        h.run(100)
        runs = []
        for _ in range(7):
            t0 = time.perf_counter()
            h.run(20)
            runs.append(time.perf_counter() - t0)
        t.append(np.median(runs))
    assert t[0] < 1.05 * t[1], t
