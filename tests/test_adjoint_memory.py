"""GPU: an adjoint handle whose allocation fails (the device's memory is held
by another allocation meanwhile) refuses to evaluate with the parameters it
could not hold, and works as a fresh one once they fit."""
import contextlib
import dataclasses

import numpy as np
import pytest

from test_adjoint_sizes import system

pytestmark = pytest.mark.gpu

MIB = 1 << 20


@contextlib.contextmanager
def device_memory_left(size):
    """All but about `size` bytes of the device's free memory are taken."""
    import torch
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    hold = torch.empty(free - size, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del hold
        torch.cuda.empty_cache()


def code(abi, call):
    with pytest.raises(abi.CvrError) as e:
        call()
    return e.value.code


def params(a, s):
    a.set_params(s.charge, s.epsilon, s.sigma, s.rc_lj, s.alpha, s.rc_r, s.kmax, s.k_e, s.dt)


@pytest.mark.parametrize("prec", [0, 1])
def test_parameters_that_do_not_fit(cuda_lib, prec):
    small = system(20000, 2, kmax=1)
    large = dataclasses.replace(small, kmax=10)  # 54 MB of chunk sums and tables or more
    a = cuda_lib.Adjoint.from_system(small, prec)
    a.forces()
    with device_memory_left(24 * MIB):
        for _ in range(2):
            assert code(cuda_lib, lambda: params(a, large)) == 7
            assert code(cuda_lib, a.forces) == 4
            assert code(cuda_lib, lambda: a.loss_grad(2, 1)) == 4
    params(a, large)
    fresh = cuda_lib.Adjoint.from_system(large, prec)
    for x, y in zip(a.forces()[:2], fresh.forces()[:2]):
        assert np.array_equal(x, y)


def test_checkpoints_that_do_not_fit(cuda_lib):
    s = system(20000, 2, kmax=1)
    a = cuda_lib.Adjoint.from_system(s, 0)
    a.loss_grad(2, 2)
    with device_memory_left(8 * MIB):
        for _ in range(2):
            assert code(cuda_lib, lambda: a.loss_grad(60, 1)) == 7
            assert code(cuda_lib, lambda: a.loss_grad(40, 2)) == 7  # would fit what was asked for before
    J, g = a.loss_grad(4, 2)
    J1, g1 = cuda_lib.Adjoint.from_system(s, 0).loss_grad(4, 2)
    assert J == J1
    for k in g:
        assert np.array_equal(g[k], g1[k])
