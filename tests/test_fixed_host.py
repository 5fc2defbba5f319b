"""The fixed-point DOP853 step (st_fixed.cuh) on the host, without a GPU, against
the same step in binary128 (tests/fixed_host.cpp): over static, strongly varying
and pulsed fields, rotation angles from 1e-3 to 0.4 rad, loose and tight
tolerances and spins of other norms, its spin error and the error of its step
controller's err^(-1/8) are no larger than those of the FP64 step on the same
inputs, and its accept decisions are binary128's."""
from __future__ import annotations

import platform
import shutil
import subprocess

import pytest

from conftest import REPO


@pytest.fixture(scope="module")
def fixed_host(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    exe = tmp_path_factory.mktemp("fixed") / "fixed_host"
    cmd = [cxx, "-O2", "-std=gnu++17", "-ffp-contract=off", f"-I{REPO / 'spin-tracking_gb300' / 'csrc'}",
           str(REPO / "tests" / "fixed_host.cpp"), "-o", str(exe)]
    if platform.machine() in ("x86_64", "i686", "i386"):
        cmd.append("-lquadmath")
    subprocess.run(cmd, check=True, capture_output=True, text=True)
    return exe


@pytest.mark.parametrize("norm", [1.0, 0.7, 16.0])
@pytest.mark.parametrize("rtol", [1e-12, 1e-6])
@pytest.mark.parametrize("angle", [1e-3, 0.05, 0.13, 0.4])
@pytest.mark.parametrize("kind", [0, 1, 2], ids=["static", "varying", "pulse"])
def test_step_error_is_no_larger_than_fp64(fixed_host, kind, angle, rtol, norm):
    out = subprocess.run([str(fixed_host), "20000", "7", str(kind), str(angle), str(rtol), str(norm)], check=True,
                         capture_output=True, text=True).stdout.split()
    r = dict(zip(out[::2], map(float, out[1::2])))
    assert r["taken"] >= 0.5 * 20000 and (r["refused"] == 0 or kind == 2)
    assert r["wrong"] == 0
    assert r["spin_fixed"] <= r["spin_fp64"]
    if r["judged"] >= 100:  # a median of fewer says nothing
        assert r["root8_fixed"] <= max(r["root8_fp64"], 2.0 ** -48)
