"""The fixed-point steps (st_fixed.cuh) on the host where the field lies along an axis and spin and adjoint along
or across it (tests/aligned_host.cpp): each component of the new spin, the step's error, the adjoint and the
gradient's moments is no further from binary128 than the FP64 form's on the same inputs, small components
among them, for each axis, parts of 1e-7 to 0.3 beside the axis, and a pulse of that size."""
from __future__ import annotations

import platform
import shutil
import subprocess

import pytest

from conftest import REPO

SMALL = [0.3, 0.15, 1e-2, 1e-3, 1e-5, 1e-7]
GEOMETRY = {"any": 0, "along": 1, "across": 2}


@pytest.fixture(scope="module")
def aligned_host(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    exe = tmp_path_factory.mktemp("aligned") / "aligned_host"
    cmd = [cxx, "-O2", "-std=gnu++17", "-ffp-contract=off", f"-I{REPO / 'spin-tracking_gb300' / 'csrc'}", f"-I{REPO / 'tests'}",
           str(REPO / "tests" / "aligned_host.cpp"), "-o", str(exe)]
    if platform.machine() in ("x86_64", "i686", "i386"):
        cmd.append("-lquadmath")
    subprocess.run(cmd, check=True, capture_output=True, text=True)
    return exe


def check(exe, form, spin, adjoint, small, angle, axis, pulse, field=611.4, w=6283.185307179586, least=1000):
    out = subprocess.run([str(exe), str(form), "1500", "11", str(GEOMETRY[spin]), str(GEOMETRY[adjoint]), str(small), str(angle),
                          str(axis), str(pulse), str(field), str(w)], check=True, capture_output=True, text=True).stdout.strip().splitlines()
    head = out[0].split()
    assert int(head[1]) >= least and int(head[5]) == 0, head
    if int(head[7]) >= 100:  # the medians of err^(-1/8)'s relative error
        assert float(head[9]) <= float(head[10])
    for line in out[1:]:
        part, fixed, fp64 = line.split()
        assert float(fixed) <= float(fp64), (part, fixed, fp64)


@pytest.mark.parametrize("axis,pulse", [(0, 0), (0, 1), (1, 0), (2, 1)])
@pytest.mark.parametrize("small", SMALL)
@pytest.mark.parametrize("spin", sorted(GEOMETRY))
@pytest.mark.parametrize("form", [0, 2, 3], ids=["dop853", "rk45q", "rkf45q"])
def test_steps(aligned_host, form, spin, small, axis, pulse):
    for angle in (0.003, 0.13):
        check(aligned_host, form, spin, "any", small, angle, axis, pulse)


@pytest.mark.parametrize("axis,pulse", [(0, 0), (0, 1), (1, 0), (2, 1)])
@pytest.mark.parametrize("small", SMALL)
@pytest.mark.parametrize("adjoint", sorted(GEOMETRY))
@pytest.mark.parametrize("spin", sorted(GEOMETRY))
def test_step_adjoint(aligned_host, spin, adjoint, small, axis, pulse):
    for angle in (0.003, 0.05, 0.16):
        check(aligned_host, 1, spin, adjoint, small, angle, axis, pulse)


@pytest.mark.parametrize("spin", sorted(GEOMETRY))
@pytest.mark.parametrize("small", [0.3, 1e-3])
@pytest.mark.parametrize("angle", [0.7, 1.0, 1.8, 2.6])
@pytest.mark.parametrize("form", [2, 3], ids=["rk45q", "rkf45q"])
def test_rotations_of_radians_in_a_pulse(aligned_host, form, angle, small, spin):
    """In a strong field a step of radians is short against the pulse's quarter turn, so that it is taken."""
    check(aligned_host, form, spin, "any", small, angle, 0, 1, field=3e5)


@pytest.mark.parametrize("spin", ["along", "across"])
@pytest.mark.parametrize("w", [1e5, 6e5, 3e6])
@pytest.mark.parametrize("form", [0, 1, 2, 3], ids=["dop853", "adjoint", "rk45q", "rkf45q"])
def test_turns_of_the_pulse_in_a_step(aligned_host, form, w, spin):
    """Steps of up to 16 turns of a weak fast pulse.  (The stages of DOP853 do not resolve it above a turn or so: its
    sums leave their range for most of them, which FP64 takes.)"""
    check(aligned_host, form, spin, spin, 1e-2, 0.01, 0, 1, w=w, least=10 if w > 1e6 and form < 2 else 700)
