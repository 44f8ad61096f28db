"""GPU: runs of small short-range systems, whose steps share one launch, against
the one-kernel-per-stage path (taken while kernel timing is on, and itself
checked against the reference elsewhere): the same functions per atom, so
positions, velocities, accelerations, thermo records and build counts must be
equal bit for bit, at sizes around a block, a warp per atom and four atoms per
warp; with a thermostat, whose kinetic energy is summed in another order, to
1e-10 of the velocities after 25 steps (1e-14 per step, times the steps, times
the growth of a perturbation over 0.125 time units, below 10)."""
import dataclasses

import numpy as np
import pytest

from caviar_b200 import workloads as W

pytestmark = pytest.mark.gpu


def system(n, kind="lj", seed=3):
    cells = next(c for c in range(3, 40) if 4 * c ** 3 >= n)
    s = W.fcc_lattice(cells, 0.8442, 0.9, seed, jitter=0.05)
    rng = np.random.default_rng(seed)
    keep = np.sort(rng.permutation(s.n)[:n])
    s = dataclasses.replace(s, pos=s.pos[keep], vel=s.vel[keep], type=s.type[keep])
    if kind == "lj":
        return s
    s.mass, s.charge = np.array([1.0, 2.0]), np.zeros(2)
    s.type = rng.integers(0, 2, n).astype(np.int32)
    s.lj = W.LJParams(2.5, np.array([[1.0, 0.75], [0.75, 0.5]]), np.array([[1.0, 0.94], [0.94, 0.88]]))
    if kind == "molecules":
        s.lj.ignore_intra_molecule = True
        s.mol = (np.arange(n) // 3).astype(np.int32)
    if kind == "stretched":  # no fixed-point displacements
        s.hi = s.hi * np.array([1.0, 1.0, 1.25])
        s.pos = s.pos * np.array([1.0, 1.0, 1.25])
    if kind == "open":
        s.bc = (1, 0, 1)
    return s


def both(abi, s, prec, steps, every, policy=0, setup=lambda sim: None):
    out = []
    for staged in (False, True):
        sim = abi.Simulation(s, precision=prec, policy=policy)
        setup(sim)
        sim.set_kernel_timing(staged)
        th = [sim.run(k, every) for k in steps]
        out.append((*sim.state(), np.concatenate(th), sim.info()["builds"]))
        sim.close()
    return out


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n", [1, 33, 127, 4144, 4145, 20001])
def test_sizes(cuda_lib, n, prec):
    a, b = both(cuda_lib, system(n), prec, [1, 24], 8)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
    assert n < 100 or a[4] > 2


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("kind", ["mixture", "molecules", "stretched", "open"])
@pytest.mark.parametrize("n", [700, 6001])
def test_forms(cuda_lib, kind, n, prec):
    a, b = both(cuda_lib, system(n, kind), prec, [25], 5)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("policy", [1, 2])
@pytest.mark.parametrize("every", [0, 1])
def test_policies_and_records(cuda_lib, policy, every):
    a, b = both(cuda_lib, system(500), 0, [7, 1, 12], every, policy)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("kind", ["berendsen", "nose_hoover"])
@pytest.mark.parametrize("n", [500, 6001])
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


def test_failed_run_leaves_the_context_usable(cuda_lib):
    s = system(500)
    sim = cuda_lib.Simulation(s, precision=0)
    bad = s.pos.copy()
    bad[7] = bad[8]  # coincident atoms: an infinite force
    sim.set_state(bad, s.vel, s.type)
    with pytest.raises(cuda_lib.CvrError):
        sim.run(20)
    sim.set_state(s.pos, s.vel, s.type)
    sim.run(20)
    fresh = cuda_lib.Simulation(s, precision=0)
    fresh.run(20)
    for x, y in zip(sim.state(), fresh.state()):
        assert np.array_equal(x, y)
