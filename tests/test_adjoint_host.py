"""The fixed-point DOP853 step adjoint (st_fixed.cuh) on the host, without a GPU, against
the same in binary128 (tests/adjoint_host.cpp): over static, strongly varying and
pulsed fields, rotation angles from 1e-4 to 0.6 rad (the scale of the stage adjoints
changes at each power of two) and other norms, the largest errors of the adjoint and
of the gradient moments are no larger than those of the FP64 form on the same inputs."""
from __future__ import annotations

import platform
import shutil
import subprocess

import pytest

from conftest import REPO


@pytest.fixture(scope="module")
def adjoint_host(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    exe = tmp_path_factory.mktemp("adjoint") / "adjoint_host"
    cmd = [cxx, "-O2", "-std=gnu++17", "-ffp-contract=off", f"-I{REPO / 'spin-tracking_gb300' / 'csrc'}",
           str(REPO / "tests" / "adjoint_host.cpp"), "-o", str(exe)]
    if platform.machine() in ("x86_64", "i686", "i386"):
        cmd.append("-lquadmath")
    subprocess.run(cmd, check=True, capture_output=True, text=True)
    return exe


@pytest.mark.parametrize("norm", [1.0, 0.7, 1e-5])
@pytest.mark.parametrize("angle", [1e-4, 0.02, 0.05, 0.13, 0.3, 0.6])
@pytest.mark.parametrize("kind", [0, 1, 2], ids=["static", "varying", "pulse"])
def test_step_adjoint_error_is_no_larger_than_fp64(adjoint_host, kind, angle, norm):
    out = subprocess.run([str(adjoint_host), "4000", "7", str(kind), str(angle), str(norm)], check=True, capture_output=True,
                         text=True).stdout.split()
    r = dict(zip(out[::2], map(float, out[1::2])))
    assert r["taken"] >= 1000
    assert r["lam_fixed"] <= r["lam_fp64"]
    assert r["mom_fixed"] <= r["mom_fp64"]
