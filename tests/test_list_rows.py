"""GPU: the list searches' pair sets against the oracle's, equal as sets, where
a stencil row's contiguous range holds from under one to over three words of 32
candidates, in boxes with and without a wrap and narrower than the stencil."""
import dataclasses

import numpy as np
import pytest

from caviar_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bc", [(1, 1, 1), (0, 1, 0)])
@pytest.mark.parametrize("density", [0.5, 2.2, 5.0, 9.0])
@pytest.mark.parametrize("n", [33, 1201, 4000])
def test_pairs(cuda_lib, oracle_lib, n, density, bc):
    s = W.fcc_lattice(10, density, 0.7, 4, jitter=0.2)
    scale = np.cbrt(n / s.n)
    rng = np.random.default_rng(n)
    keep = np.sort(rng.permutation(s.n)[:n])
    s = dataclasses.replace(s, pos=s.pos[keep] * scale, vel=s.vel[keep], type=s.type[keep])
    s.lo, s.hi, s.bc = s.lo * scale, s.hi * scale, bc
    o = oracle_lib.Oracle(s)
    o.setup()
    ref = o.pairs()
    for kind in (cuda_lib.LIST_THREAD, cuda_lib.LIST_WARP):
        for prec in (cuda_lib.PREC_FP64, cuda_lib.PREC_MIXED):
            sim = cuda_lib.Simulation(s, precision=prec, list_kernel=kind)
            sim.build_neighbors(True)
            assert np.array_equal(sim.pairs(), ref)
            sim.close()
