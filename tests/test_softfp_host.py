"""The trajectory's integer division, square root, uniform draws and comparisons
(st_softfp.cuh) on the host against the host's correctly rounded operations
(tests/softfp_host.cpp): every result equal bit for bit, special values included."""
from __future__ import annotations

import shutil
import subprocess

import pytest

from conftest import REPO


@pytest.mark.parametrize("seed", [1, 2])
def test_equal_to_ieee(tmp_path, seed):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    exe = tmp_path / "softfp_host"
    subprocess.run([cxx, "-O2", "-std=gnu++17", "-ffp-contract=off", f"-I{REPO / 'spin-tracking_gb300' / 'csrc'}",
                    str(REPO / "tests" / "softfp_host.cpp"), "-o", str(exe)], check=True, capture_output=True, text=True)
    out = subprocess.run([str(exe), "1000000", str(seed)], check=True, capture_output=True, text=True).stdout.split()
    assert dict(zip(out[::2], map(int, out[1::2]))) == {"div": 0, "sqrt": 0, "unit": 0, "compare": 0}
