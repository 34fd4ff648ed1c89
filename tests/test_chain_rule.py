"""Chained launches (csrc/chain.cuh): a chained kernel starts while the kernel before it still
stores, so its field pointers must not be __restrict__ (a promise that the data is read-only for
the kernel's lifetime, which lets loads move above the wait or take the non-coherent path)."""
import math
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mcstar-libs_b200", "csrc")
TABLES = {"tw", "twg", "tab", "post"}  # written by pfc_create alone
CHAINED = {"k_cols", "k_rows", "k_xpass", "k_zprop", "k_ycol", "k_xrow", "k_zcol", "k_zcarry"}


def _sources():
    return {f: open(os.path.join(CSRC, f)).read() for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh"))}


def _kernels():
    """name -> (parameter list, body) of every kernel that waits for the one before it."""
    out = {}
    for text in _sources().values():
        for m in re.finditer(r"__global__ void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\(([^{;]*?)\)\s*\{", text):
            body = text[m.end():]
            stop = body.find("\n}\n")
            if "chain_wait();" in body[:stop]:
                out[m.group(1)] = m.group(2)
    return out


def test_chained_kernels_promise_read_only_data_for_tables_alone():
    kernels = _kernels()
    assert CHAINED <= set(kernels)
    for name, params in kernels.items():
        promised = {p.split()[-1].lstrip("*&") for p in params.split(",") if "__restrict__" in p}
        assert promised <= TABLES, f"{name}: {sorted(promised - TABLES)}"


@pytest.mark.gpu
@pytest.mark.parametrize("options", [None, {"z_carry": 0}, {"z_carry": 1}], ids=["default", "carry-A", "carry-psi"])
@pytest.mark.parametrize("shape", [(64, 64, 64), (128, 128, 128), (60, 50, 40), (48, 40, 1)], ids=str)
def test_chained_steps_equal_separated_ones(shape, options):
    """Many short calls back to back, chained, against the same calls with an event between the
    passes (tracing), bit for bit."""
    from mcstar_b200 import Stepper
    if shape[2] == 1 and options:
        pytest.skip("2D fields have one schedule")
    nx, ny, nz = shape
    psi = (-0.2 + 0.1 * np.random.default_rng(3).uniform(-1, 1, (nz, ny, nx))).astype(np.float32)
    got = []
    for traced in (False, True):
        st = Stepper(shape, math.pi / 4, 0.5, 0.3, namp=0.02, seed=5, options=options)
        st.set_real(psi)
        st.ctx.profile_enable(traced)
        for n in [1] * 40 + [2, 3, 30]:
            st.step(n)
        st.ctx.profile_enable(False)
        got.append(st.kspace())
    assert np.array_equal(got[0], got[1])
