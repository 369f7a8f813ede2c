"""The FP64 reciprocals of the eliminations' pivots against the correctly rounded 1 / x.

Both start from a seed of relative error e = 2^-19.9.  Two Newton-Raphson steps (rcp_newton) leave e^4 = 2^-79.6, 2^-26 of a
unit in the last place; one third-order step (rcp_cubic) leaves e^3 = 2^-59.7, 2^-6.7 of a unit.  A result then differs
from the rounded quotient only where that lies as close as this to the middle of two numbers, by one unit: for at most
twice that share of the values if every seed had the largest error, 3e-8 and 2e-2, bounded here by 1e-6 and 2e-2."""
import ctypes

import numpy as np
import pytest

from harness import build


@pytest.mark.gpu
@pytest.mark.parametrize("order,share", [(2, 1e-6), (3, 2e-2)])
def test_reciprocal_is_the_rounded_quotient(tmp_path, order, share):
    import torch
    lib = build(tmp_path)
    rng = np.random.default_rng(5)
    n = 1 << 22
    x = np.ldexp(1.0 + rng.random(n), rng.integers(-250, 251, n))
    x[:501] = np.ldexp(1.0, np.arange(-250, 251))
    d = torch.as_tensor(x, device="cuda")
    r = torch.empty_like(d)
    torch.cuda.synchronize()
    assert lib.stage_rcp(n, order, ctypes.c_void_p(d.data_ptr()), ctypes.c_void_p(r.data_ptr())) == 0
    ulps = np.abs(r.cpu().numpy().view(np.int64) - (1.0 / x).view(np.int64))
    assert ulps.max() <= 1 and (ulps > 0).mean() <= share, (ulps.max(), (ulps > 0).mean())
