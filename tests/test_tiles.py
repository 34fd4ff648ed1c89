"""Column passes of fields with few columns use the multiprocessors they can: with columns to spread, no
pass is left with fewer CTAs than half of them (on the CPU, over the plans)."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT, build_shim_driver


@pytest.mark.skipif(shutil.which("nvcc") is None and not os.path.exists("/usr/local/cuda/bin/nvcc"),
                    reason="nvcc not available")
def test_few_columns_are_spread(tmp_path):
    exe = tmp_path / "driver_tiles"
    rc, out = build_shim_driver("float", exe, os.path.join(ROOT, "tests", "plan", "driver_tiles.cu"))
    assert rc == 0, out
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0
    lines = r.stdout.splitlines()
    assert not [s for s in lines if s.startswith("bad")], "\n".join(lines[:20])
    assert int(lines[-1].split()[1]) > 1000
