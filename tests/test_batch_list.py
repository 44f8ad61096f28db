"""GPU: replicas around the size from which the batch takes LJ pair lists, with
no and some atoms charged, several LJ types, a list that overflows (the
all-pairs form stands in), and a run over several rebuilds; against the FP64
replica oracle with the tolerances of tests/test_batch.py."""
import numpy as np
import pytest

from caviar_b200 import workloads as W
from helpers import force_errors
from test_batch import ENERGY_TOL, FORCE_TOL, MAX_TOL, make_batch, oracle_forces, replica

pytestmark = pytest.mark.gpu


def batch(sizes, charges="mixed", density=0.8, types=False):
    b = W.replica_batch(sizes=sizes, seed=21, density=density)
    rng = np.random.default_rng(2)
    n = len(b.type)
    if charges == "none":
        b.type = np.zeros(n, np.int32)
    if types:
        e = np.array([1.0, 0.8, 0.5])
        b.epsilon = np.sqrt(np.outer(e, e))
        b.sigma = 0.5 * (np.array([1.0, 0.9, 0.8])[:, None] + np.array([1.0, 0.9, 0.8]))
    if density > 1:  # dense: smaller atoms, more of them within the cutoff
        b.sigma = b.sigma * 0.55
    return b


@pytest.mark.parametrize("charges,density,types", [("none", 0.8, False), ("mixed", 0.8, True), ("mixed", 3.0, False)])
def test_forces_and_energies(cuda_lib, oracle_lib, charges, density, types):
    b = batch([191, 192, 193, 257, 700], charges, density, types)
    h = make_batch(cuda_lib, b)
    out = h.run(0)
    acc = h.state()[2]
    for r in range(len(b.n)):
        ref, en = oracle_forces(oracle_lib, b, r)
        g, m, _ = force_errors(acc[replica(b, r)], ref)
        assert g < FORCE_TOL and m < MAX_TOL, (b.n[r], g, m)
        got = dict(zip(h.OUT_KEYS, out[r]))
        for k in ("e_lj", "e_ewald_r", "virial"):
            assert abs(got[k] - en[k]) <= ENERGY_TOL * max(1.0, abs(en[k])), (b.n[r], k)


def test_run_over_rebuilds(cuda_lib, oracle_lib):
    b = batch([200, 450])
    h = make_batch(cuda_lib, b)
    h.run(40)
    pos, vel, _ = h.state()
    for r in range(2):
        sl = replica(b, r)
        L = float(b.box[r])
        p, v, _ = oracle_lib.replica_run(int(b.n[r]), b.pos[sl], b.vel[sl], b.type[sl], L, b.mass, b.charge, b.epsilon,
                                         b.sigma, float(b.rc_lj[r]), b.alpha, float(b.rc_r[r]), b.kmax, b.k_e, b.dt, 40)
        d = pos[sl] - p
        assert np.abs(d - L * np.round(d / L)).max() < 1e-6
        assert np.abs(vel[sl] - v).max() < 1e-4
