"""The update divides by D(k): modes of an FP32 field whose D lies between 2^126 (where an
approximate reciprocal is zero) and the largest float have their value."""
import math

import numpy as np
import pytest

import pfc_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(24, 20, 12), (24, 20, 1)], ids=str)
def test_large_denominators(shape):
    """dt is such that the largest D is 2e38.  The modes compared carry the nonlinear term's transform,
    a few thousandths of its largest mode: FP32 gives them to 1e-4."""
    from mcstar_b200 import Stepper
    nx, ny, nz = shape
    dx, eps, C = math.pi / 4, 0.3, 1.0
    k1 = [2 * math.pi * np.fft.fftfreq(n, dx) for n in (nz, ny)] + [2 * math.pi * np.fft.rfftfreq(nx, dx)]
    k2 = k1[0][:, None, None] ** 2 + k1[1][None, :, None] ** 2 + k1[2][None, None, :] ** 2
    growth = k2 * (1 + C - eps - 2 * k2 + k2 * k2)
    dt = 2e38 / growth.max()
    k0 = O.r2c(-0.2 + 0.1 * np.random.default_rng(9).uniform(-1, 1, (nz, ny, nx)))
    st = Stepper(shape, dx, dt, eps, dtype=np.float32)
    st.set_kspace(k0.astype(np.complex64))
    st.step(1)
    want = O.step(k0, 1, dt, eps, st.lens, shape)
    large = dt * growth > 1.01 * 2.0 ** 126
    assert large.sum() > 5
    err = np.linalg.norm(st.kspace()[large] - want[large]) / np.linalg.norm(want[large])
    assert err < 1e-3
