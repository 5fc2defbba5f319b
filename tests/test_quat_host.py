"""The fixed-point quaternion steps (st_fixed.cuh) on the host, without a GPU, against the
same steps in binary128 (tests/quat_host.cpp): over static, strongly varying and
pulsed fields, rotation angles from 1e-7 to 3 rad and spins of other norms, the largest
errors of their proposals and error vectors are no larger than those of the
FP64 steps on the same inputs."""
from __future__ import annotations

import platform
import shutil
import subprocess

import pytest

from conftest import REPO


@pytest.fixture(scope="module")
def quat_host(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    exe = tmp_path_factory.mktemp("quat") / "quat_host"
    cmd = [cxx, "-O2", "-std=gnu++17", "-ffp-contract=off", f"-I{REPO / 'spin-tracking_gb300' / 'csrc'}",
           str(REPO / "tests" / "quat_host.cpp"), "-o", str(exe)]
    if platform.machine() in ("x86_64", "i686", "i386"):
        cmd.append("-lquadmath")
    subprocess.run(cmd, check=True, capture_output=True, text=True)
    return exe


@pytest.mark.parametrize("stepper", [0, 1], ids=["rk45q", "rkf45q"])
@pytest.mark.parametrize("norm", [1.0, 0.7])
@pytest.mark.parametrize("angle", [1e-7, 1e-4, 0.01, 0.4, 1.0, 2.6])
@pytest.mark.parametrize("kind", [0, 1, 2], ids=["static", "varying", "pulse"])
def test_step_error_is_no_larger_than_fp64(quat_host, kind, angle, norm, stepper):
    out = subprocess.run([str(quat_host), "4000", "7", str(kind), str(angle), str(norm), str(stepper)], check=True, capture_output=True,
                         text=True).stdout.split()
    r = dict(zip(out[::2], map(float, out[1::2])))
    # the long segments' varying fields grow past 4 rad a step, long pulsed steps pass a quarter turn of the pulse
    assert r["taken"] >= (0.5 * 4000 if kind == 0 or angle <= 0.4 else 1000 if kind == 1 else 0)
    assert r["spin_fixed"] <= r["spin_fp64"]
    assert r["err_fixed"] <= r["err_fp64"]
