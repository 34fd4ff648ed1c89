"""The general-length passes (csrc/genfft.cuh): plain transforms and steps at the lengths where
the engine's stages, padding and tiles can go wrong -- prime radices (with the appended stage of
radix 1), odd and even last radices, one to five stages, odd row lengths (a last unpaired row in
FP32), partial last column tiles, one-mode-wide fields -- against numpy in FP64.

Tolerances: a transform of n points does about log2 n roundings per value, each within half
an ulp (2^-24, 2^-53) of the running value and independent: the relative L2 error stays below
log2(n) ulps with a factor to spare over its sqrt(log2 n) expectation."""
import math

import numpy as np
import pytest

import pfc_oracle as O

pytestmark = pytest.mark.gpu

F32, F64 = np.float32, np.float64
SHAPES = [(7, 5, 3), (14, 9, 1), (26, 31, 4), (2, 2, 2), (1, 6, 4), (15, 1, 1), (62, 49, 5), (30, 24, 18), (34, 27, 25),
          (66, 50, 36), (121, 100, 1), (250, 240, 3), (90, 81, 80), (400, 375, 1), (2000, 7, 1), (22, 1280, 1),
          (1458, 625, 1), (720, 36, 11)]


def rel(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


@pytest.mark.parametrize("dtype", [F32, F64], ids=["f32", "f64"])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_general_transforms(shape, dtype):
    from mcstar_b200 import C2R, R2C, CPUArray, CufftPlan, GPUArray
    nx, ny, nz = shape
    x = np.random.default_rng(5).uniform(-1, 1, (nz, ny, nx)).astype(dtype)
    want = np.fft.rfftn(x.astype(F64), axes=(0, 1, 2))
    tol = max(1.0, math.log2(x.size)) * (2.0 ** -24 if dtype == F32 else 2.0 ** -53)
    h = CPUArray(shape, dtype)
    h.numpy()[: x.size] = x.ravel()
    a, k, b = GPUArray(h), GPUArray(shape, dtype), GPUArray(shape, dtype)
    CufftPlan(dtype, R2C, shape).execute(a, k)
    assert rel(k.ptr_cmpl().cpu().numpy(), want) < tol
    CufftPlan(dtype, C2R, shape).execute(k, b)
    assert rel(b.ptr_real().cpu().numpy() / x.size, x) < 2 * tol


STEPS = [((121, 100, 1), F32), ((15, 1, 1), F64), ((400, 375, 1), F64), ((34, 27, 25), F32), ((66, 50, 36), F64),
         ((62, 49, 5), F32), ((96, 96, 96), F32)]


@pytest.mark.parametrize("shape,dtype", STEPS, ids=str)
def test_general_steps_and_resume(shape, dtype):
    """Steps with noise against the oracle, and a run cut in two repeating its bits (the entry
    transform of a call is the inverse transform of the step before it)."""
    from mcstar_b200 import Stepper
    nx, ny, nz = shape
    psi = -0.2 + 0.1 * np.random.default_rng(6).uniform(-1, 1, (nz, ny, nx))
    k0 = O.r2c(psi)
    runs = []
    for cuts in ((5,), (2, 3)):
        st = Stepper(shape, math.pi / 4, 0.5, 0.3, dtype=dtype, namp=0.03, seed=11)
        st.set_kspace(k0.astype(np.complex64 if dtype == F32 else np.complex128))
        for n in cuts:
            st.step(n)
        runs.append(st.kspace())
    want = O.step(k0, 5, 0.5, 0.3, st.lens, shape, namp=0.03, seed=11, noise_dtype=dtype)
    assert rel(runs[0], want) < (2e-6 if dtype == F32 else 1e-12)
    assert np.array_equal(runs[0], runs[1])
    assert runs[0][0, 0, 0] == k0.astype(runs[0].dtype)[0, 0, 0]


@pytest.mark.parametrize("shape", [(16, 16, 256), (16, 12, 256), (32, 8, 128), (48, 24, 192), (64, 64, 128)], ids=str)
def test_edge_column_tiles(shape):
    """The register z pass whose last tile is the kx = nx/2 column alone takes it at eight ky per
    CTA where 8 divides ny, and as a tile of its own elsewhere (ny = 12)."""
    from mcstar_b200 import Stepper
    nx, ny, nz = shape
    k0 = O.r2c(-0.2 + 0.1 * np.random.default_rng(9).uniform(-1, 1, (nz, ny, nx)))
    st = Stepper(shape, math.pi / 4, 0.5, 0.3, dtype=F32, namp=0.03, seed=3)
    st.set_kspace(k0.astype(np.complex64))
    st.step(4)
    want = O.step(k0, 4, 0.5, 0.3, st.lens, shape, namp=0.03, seed=3, noise_dtype=F32)
    got = st.kspace()
    assert rel(got, want) < 2e-6
    assert rel(got[..., nx // 2], want[..., nx // 2]) < 2e-5


@pytest.mark.parametrize("dtype", [F32, F64], ids=["f32", "f64"])
@pytest.mark.parametrize("shape", [(4, 4, 1), (8, 6, 5), (10, 3, 1), (36, 5, 1), (54, 7, 3), (50, 11, 2), (90, 9, 1),
                                   (72, 30, 4), (2400, 3, 1)], ids=str)
def test_paired_x_pass(shape, dtype):
    """The x pass that splits and merges the real transforms in the first stage's registers: first
    radices 2 to 5, odd and even numbers of its butterflies (the middle one pairs with itself),
    an appended stage of radix 1, an unpaired last row in FP32."""
    from mcstar_b200 import Stepper
    nx, ny, nz = shape
    k0 = O.r2c(-0.2 + 0.1 * np.random.default_rng(4).uniform(-1, 1, (nz, ny, nx)))
    st = Stepper(shape, math.pi / 4, 0.25, 0.3, dtype=dtype)
    st.set_kspace(k0.astype(np.complex64 if dtype == F32 else np.complex128))
    st.step(3)
    want = O.step(k0, 3, 0.25, 0.3, st.lens, shape)
    assert rel(st.kspace(), want) < (2e-6 if dtype == F32 else 1e-12)


@pytest.mark.parametrize("n,box,rlim", [(1, 50.0, 5.0), (2, 50.0, 40.0), (33, 30.0, 8.0), (150, 12.0, 12.0),
                                        (700, 40.0, 12.5), (900, 64.0, 9.0)])
def test_bond_order_lists(n, box, rlim):
    """Bond order at the neighbour lists' edges: no neighbours, all pairs (fewer than three cells per
    side), lists beyond the 96 entries a warp sorts in shared memory, several blocks of rows."""
    from mcstar_b200 import Context, maximum_dtype
    import torch
    rng = np.random.default_rng(n)
    idx = rng.uniform(0, box, (n, 3)).astype(F32)
    field = rng.uniform(-0.1, 1.0, n).astype(F32)
    M = np.zeros(n, dtype=maximum_dtype(F32))
    M["i0"], M["i1"], M["i2"], M["field"] = idx[:, 0], idx[:, 1], idx[:, 2], field
    ctx = Context((8, 8, 8), F32)
    dev = torch.from_numpy(M.view(np.uint8).ravel().copy()).cuda()
    rows = ctx.bond_order(dev, n, (1.0, 1.0, 1.0), 0.0, box, rlim).cpu().numpy()
    res, _ = O.bond_order(idx, field, (1.0, 1.0, 1.0), 0.0, box, rlim)
    assert rows.shape[0] == len(res["x"])
    for i, c in enumerate(O.BOND_COLUMNS):
        np.testing.assert_allclose(rows[:, i], res[c], atol=1e-9, rtol=1e-9, err_msg=c)


def test_status_words_between_calls():
    """The stepper clears its status words only after a call that found one set: a bad state is
    reported by the call that meets it and by no later one, however good and bad calls alternate."""
    from mcstar_b200 import PfcError
    from test_gpu_step import stepper
    shape = (48, 40, 1)
    psi = -0.2 + 0.05 * np.random.default_rng(2).uniform(-1, 1, shape[::-1])
    st = stepper(shape, F32)
    for bad in (False, False, True, True, False, True, False, False):
        st.set_real(psi)
        if bad:
            st.kpsi[10] = float("nan")
            with pytest.raises(PfcError):
                st.step(1)
        else:
            st.step(1)
            assert np.isfinite(st.real()).all()


@pytest.mark.parametrize("dtype", [F32, F64], ids=["f32", "f64"])
@pytest.mark.parametrize("shape", [(24, 20, 1), (20, 18, 12)], ids=str)
def test_nonfinite_parameters_are_reported(shape, dtype):
    """A NaN in the propagator reaches the new state, and the call reports it."""
    from mcstar_b200 import PfcError
    from test_gpu_step import stepper
    st = stepper(shape, dtype, eps=float("nan"))
    st.set_real(-0.2 + 0.05 * np.random.default_rng(2).uniform(-1, 1, shape[::-1]))
    with pytest.raises(PfcError):
        st.step(2)
