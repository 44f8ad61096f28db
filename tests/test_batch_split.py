"""GPU: a run of a replica batch split over two calls is bit-identical to one
run also where the LJ list of a replica overflows at its first build and would
fit a few steps later: clusters of 300 atoms that expand, whose fullest row
drops below the list's capacity (128) between the second and the eighth step."""
import numpy as np
import pytest

from caviar_b200 import workloads as W
from test_batch import make_batch

pytestmark = pytest.mark.gpu

STEPS = 10


@pytest.mark.parametrize("spacing", [0.84, 0.86, 0.88])
def test_split_runs(cuda_lib, spacing):
    b = W.replica_batch(sizes=[300], density=300 / 12.0 ** 3)
    g = np.arange(7) - 3.0
    sites = np.stack(np.meshgrid(g, g, g, indexing="ij"), axis=-1).reshape(-1, 3)[:300]
    x = spacing * sites + np.random.default_rng(5).uniform(-0.03, 0.03, sites.shape)
    b.pos, b.vel, b.type = x + 6.0, 1.6 * x, np.zeros(300, np.int32)
    b.sigma = 0.55 * b.sigma
    h = make_batch(cuda_lib, b)
    h.run(STEPS)
    one = h.state()
    for k in range(1, STEPS):
        h.set_state(b.pos, b.vel, b.type)
        h.run(k)
        h.run(STEPS - k)
        for p, q in zip(one, h.state()):
            assert np.array_equal(p, q), k
