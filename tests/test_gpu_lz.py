"""The height of a 2D field: any length gives kz = 0; one that gives no number (0, NaN) is reported as
a non-finite state, as pfc_update_eom and the energy have it."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64], ids=["f32", "f64"])
@pytest.mark.parametrize("shape", [(24, 20, 1), (128, 128, 1), (15, 1, 1)], ids=str)
def test_height_of_a_film(shape, dtype):
    from mcstar_b200 import Context, PfcError
    ctx = Context(shape, dtype)
    lens = [n * 0.8 for n in shape]
    out = []
    for lz in (0.8, 1e3, math.inf, 0.0, math.nan):
        k = ctx.empty_state()
        k.zero_()
        k[0] = -0.2 * ctx.n_real
        k[2] = 0.1 * ctx.n_real / 2
        call = lambda: ctx.step(k, 2, 0.5, 0.3, (lens[0], lens[1], lz))
        if lz > 0.0:
            call()
            out.append(k.cpu().numpy())
        else:
            with pytest.raises(PfcError):
                call()
    assert np.isfinite(out[0]).all()
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
