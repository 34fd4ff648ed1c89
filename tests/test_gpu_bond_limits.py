"""Neighbour radii at the ends of their range: an atom without a position (infinite coordinate) has no
neighbours at any finite radius, and every other pair is one from the box's diagonal up."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64], ids=["f32", "f64"])
@pytest.mark.parametrize("rlim", [1e-200, 1e-120, 60.0, 1e149, 1e151, 1e200, 1.7e308])
def test_extreme_radii(rlim, dtype):
    import torch
    from mcstar_b200 import Context, maximum_dtype
    n, box = 40, 30.0
    x = np.random.default_rng(1).uniform(0, box, (n, 3)).astype(dtype)
    x[3, 1] = math.inf
    M = np.zeros(n, dtype=maximum_dtype(dtype))
    M["i0"], M["i1"], M["i2"], M["field"] = x[:, 0], x[:, 1], x[:, 2], 1.0
    ctx = Context((8, 8, 8), dtype)
    dev = torch.from_numpy(M.view(np.uint8).ravel().copy()).cuda()
    rows = ctx.bond_order(dev, n, (1.0, 1.0, 1.0), 0.0, box, rlim).cpu().numpy()
    if rlim < 1.0:
        assert rows.shape[0] == 0
    else:
        assert rows.shape[0] == n - 1
        assert (rows[:, 3] == n - 2).all()
