"""GPU: sizes at the edges of the allocation-free structure factor's split
(k-set shapes that fill one or several blocks and m-groups, atom counts around
the smallest chunk and the shared-memory stage) against a direct FP64 sum.

Tolerance: each term's phase is rounded to about (2 pi k_max + 10) 2^-53 per
axis on either side, so |dS| <= 3 (2 pi 30 + 10) 2 * 1.2e-16 sum |q| < 2e-13 sum |q|
for every k_max up to 30, whatever the order of the sum.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def direct(pos, q, box, kmax):
    kx, ky, kz = kmax
    g = np.stack(np.meshgrid(*[np.arange(-k, k + 1) for k in kmax], indexing="ij"), axis=-1).reshape(-1, 3)
    g = g[np.any(g != 0, axis=1)][: 8 * kx * ky * kz]
    e = [np.exp(2j * np.pi * np.outer(np.arange(-k, k + 1), pos[:, d] / box[d])) for d, k in enumerate(kmax)]
    return np.array([np.sum(q * e[0][a + kx] * e[1][b + ky] * e[2][c + kz]) for a, b, c in g])


@pytest.mark.parametrize("kmax", [(1, 1, 1), (2, 3, 1), (1, 2, 30), (5, 4, 6), (8, 8, 8), (10, 3, 11)])
@pytest.mark.parametrize("n", [1, 31, 33, 1000, 9001])
def test_structure_factor_sizes(cuda_lib, kmax, n):
    import torch
    f = cuda_lib.load().cvr_structure_factor_noalloc
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int64, ctypes.POINTER(ctypes.c_double), ctypes.c_int,
                  ctypes.c_int, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_char_p, ctypes.c_size_t]
    f.restype = ctypes.c_int
    rng = np.random.default_rng(n)
    box = np.array([11.0, 17.0, 13.0])
    pos = rng.uniform(-0.5, 1.5, size=(n, 3)) * box
    q = rng.normal(size=n)
    nk = 8 * kmax[0] * kmax[1] * kmax[2]
    p, qd = torch.from_numpy(pos).cuda(), torch.from_numpy(q).cuda()
    out = torch.full((nk + 1, 2), float("nan"), dtype=torch.float64, device="cuda")
    rc = f(p.data_ptr(), qd.data_ptr(), n, (ctypes.c_double * 3)(*box), *kmax, out.data_ptr(),
           torch.cuda.current_stream().cuda_stream, None, 0)
    assert rc == 0
    got = out.cpu().numpy()
    assert np.isnan(got[nk]).all()  # nothing past the k-set is written
    ref = direct(pos, q, box, kmax)
    assert np.abs(got[:nk, 0] + 1j * got[:nk, 1] - ref).max() <= 2e-13 * np.abs(q).sum()
