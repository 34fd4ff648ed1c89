"""The lengths a context accepts: every one the rule of creation accepts has plans whose launches
fit a CTA's shared memory (on the CPU, over all lengths near the limit), and the long ones whose
padded lines would not fit step as the oracle does."""
import math
import os
import shutil
import subprocess

import numpy as np
import pytest

import pfc_oracle as O
from conftest import ROOT, build_shim_driver

F32, F64 = np.float32, np.float64


@pytest.mark.skipif(shutil.which("nvcc") is None and not os.path.exists("/usr/local/cuda/bin/nvcc"),
                    reason="nvcc not available")
def test_every_accepted_length_fits(tmp_path):
    exe = tmp_path / "driver_plan"
    rc, out = build_shim_driver("float", exe, os.path.join(ROOT, "tests", "plan", "driver_plan.cu"))
    assert rc == 0, out
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0
    lines = r.stdout.splitlines()
    assert not [s for s in lines if s.startswith("bad")], "\n".join(lines[:20])
    assert int(lines[-1].split()[1]) > 10000


def rel(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


@pytest.mark.gpu
@pytest.mark.parametrize("shape,options", [((16, 12288, 1), {}), ((16, 11664, 1), {}), ((5, 10240, 1), {}),
                                           ((6, 8602, 1), {}), ((24576, 4, 1), {}), ((23040, 3, 1), {}),
                                           ((6, 4, 4802), {"z_carry": 0}), ((6, 4, 6144), {"z_carry": 0}),
                                           ((6, 4, 6144), {})], ids=str)
def test_long_lines_step(shape, options):
    """FP32 steps whose lines fill a CTA's shared memory.  The tolerances are those of the general
    steps (test_gpu_general.py)."""
    from mcstar_b200 import Stepper
    nx, ny, nz = shape
    k0 = O.r2c(-0.2 + 0.1 * np.random.default_rng(2).uniform(-1, 1, (nz, ny, nx)))
    st = Stepper(shape, math.pi / 4, 0.5, 0.3, dtype=F32, namp=0.03, seed=11, options=options)
    st.set_kspace(k0.astype(np.complex64))
    st.step(3)
    want = O.step(k0, 3, 0.5, 0.3, st.lens, shape, namp=0.03, seed=11, noise_dtype=F32)
    assert rel(st.kspace(), want) < 2e-6


@pytest.mark.gpu
def test_long_lines_slab_step():
    """A field of nz = 4802 stepped as one rank's slab (the z pass that carries A)."""
    from mcstar_b200.slab import SlabRank, run_steps
    shape = (6, 4, 4802)
    nx, ny, nz = shape
    k0 = O.r2c(-0.2 + 0.1 * np.random.default_rng(2).uniform(-1, 1, (nz, ny, nx)))
    ranks = [SlabRank(shape, r, 2, math.pi / 4, 0.5, 0.3, dtype=F32, namp=0.03, seed=11) for r in range(2)]
    for r in ranks:
        r.set_kspace_slab(k0[:, r.ky0:r.ky0 + r.nys].astype(np.complex64))
    run_steps(ranks, 2)
    got = np.concatenate([r.kspace_slab() for r in ranks], axis=1)
    want = O.step(k0, 2, 0.5, 0.3, ranks[0].lens, shape, namp=0.03, seed=11, noise_dtype=F32)
    assert rel(got, want) < 2e-6


@pytest.mark.gpu
@pytest.mark.parametrize("shape,dtype", [((16, 12500, 1), F32), ((25600, 4, 1), F32), ((6, 4, 6250), F32),
                                         ((16, 6250, 1), F64), ((37, 4, 1), F32)], ids=str)
def test_refused_lengths(shape, dtype):
    from mcstar_b200 import Context, PfcError
    with pytest.raises(PfcError) as e:
        Context(shape, dtype)
    assert e.value.status == 2  # PFC_ERR_UNSUPPORTED
