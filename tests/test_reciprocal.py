"""The FP64 reciprocal of the eliminations' pivots (rcp_newton: two Newton-Raphson steps from a seed of relative error
2^-19.9) against the correctly rounded 1 / x.

The second step leaves e^4 = 2^-79 of the seed's error e, 2^-26 of a unit in the last place, so a result differs from the
rounded quotient only where that lies so close to the middle of two numbers, and then by one unit: some 2 in 10^8 values,
bounded here by 1 in 10^6."""
import ctypes

import numpy as np
import pytest

from harness import build


@pytest.mark.gpu
def test_reciprocal_is_the_rounded_quotient(tmp_path):
    import torch
    lib = build(tmp_path)
    rng = np.random.default_rng(5)
    n = 1 << 22
    x = np.ldexp(1.0 + rng.random(n), rng.integers(-250, 251, n))
    x[:501] = np.ldexp(1.0, np.arange(-250, 251))
    d = torch.as_tensor(x, device="cuda")
    r = torch.empty_like(d)
    torch.cuda.synchronize()
    assert lib.stage_rcp(n, ctypes.c_void_p(d.data_ptr()), ctypes.c_void_p(r.data_ptr())) == 0
    ulps = np.abs(r.cpu().numpy().view(np.int64) - (1.0 / x).view(np.int64))
    assert ulps.max() <= 1 and (ulps > 0).mean() <= 1e-6, (ulps.max(), (ulps > 0).mean())
