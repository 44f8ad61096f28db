"""GPU: a position or charge that is not finite reaches every k-vector of the
allocation-free structure factor, whichever axis it is on (a k-vector whose
index on that axis is 0 included)."""
import ctypes

import numpy as np
import pytest

from test_zz_no_alloc import _entry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", [0, 1, 2, "q"])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf")])
@pytest.mark.parametrize("n", [5, 3001])
def test_every_k_vector(cuda_lib, what, value, n):
    import torch
    f = _entry(cuda_lib)
    rng = np.random.default_rng(n)
    pos, q = rng.uniform(0, 9.0, size=(n, 3)), rng.normal(size=n)
    if what == "q":
        q[n // 2] = value
    else:
        pos[n // 2, what] = value
    p, qd = torch.from_numpy(pos).cuda(), torch.from_numpy(q).cuda()
    out = torch.zeros((8 * 3 * 2 * 5, 2), dtype=torch.float64, device="cuda")
    rc = f(p.data_ptr(), qd.data_ptr(), n, (ctypes.c_double * 3)(9.0, 9.0, 9.0), 3, 2, 5, out.data_ptr(),
           torch.cuda.current_stream().cuda_stream, None, 0)
    assert rc == 0
    got = out.cpu().numpy()
    if what == "q":
        assert not np.isfinite(got).any()
    else:
        assert np.isnan(got).all()
