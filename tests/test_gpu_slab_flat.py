"""The slab passes of a 2D field (nz = 1): one step through them, the update on ky-slabs of uneven
height, against the oracle."""
import ctypes
import math

import numpy as np
import pytest

import pfc_oracle as O

pytestmark = pytest.mark.gpu

F32, F64 = np.float32, np.float64


@pytest.mark.parametrize("dtype", [F32, F64], ids=["f32", "f64"])
@pytest.mark.parametrize("shape,cuts", [((48, 40, 1), (20,)), ((33, 21, 1), (1, 8)), ((1, 16, 1), ()), ((300, 7, 1), (3,))],
                         ids=str)
def test_flat_slabs_match_oracle(shape, cuts, dtype):
    import torch
    from mcstar_b200 import Context
    from mcstar_b200._lib import PfcStepParams
    nx, ny, _ = shape
    k0 = O.r2c(-0.2 + 0.1 * np.random.default_rng(2).uniform(-1, 1, (1, ny, nx)))
    lens = (nx * 0.8, ny * 0.8, 0.8)
    p = PfcStepParams(0.5, 0.3, 0.0, 1.0, 0.03, *lens, 11, 4)
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    whole = Context(shape, dtype)
    A, B = whole.empty_state(), whole.empty_state()
    A.copy_(torch.from_numpy(k0.astype(np.complex64 if dtype == F32 else np.complex128).view(dtype).ravel()))
    whole._call("pfc_slab_xy", ptr(A), ptr(B), 1.0, 0.0)
    out = []
    for lo, hi in zip((0,) + cuts, cuts + (ny,)):
        slab = Context((nx, hi - lo, 1), dtype)
        row = 2 * whole.nxh
        k, a, b = (slab.empty_state() for _ in range(3))
        k.copy_(A[lo * row:hi * row])
        b.copy_(B[lo * row:hi * row])
        slab._call("pfc_slab_zinv", ptr(k), ptr(a), lo)
        slab._call("pfc_slab_zpass", ptr(a), ptr(b), ctypes.byref(p), lo, ny, 1)
        out.append(a.cpu().numpy())
    got = np.concatenate(out).view(np.complex64 if dtype == F32 else np.complex128).reshape(1, ny, whole.nxh)
    want = O.step(k0, 1, 0.5, 0.3, lens, shape, namp=0.03, seed=11, counter0=4, noise_dtype=dtype)
    assert np.linalg.norm(got - want) < (2e-6 if dtype == F32 else 1e-12) * np.linalg.norm(want)
