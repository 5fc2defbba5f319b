"""The sanity check's |a| > b (st_softfp.cuh) on the host: the host's own result for every pair of special values,
limits below zero among them (a box edge below zero puts every position out of bounds)."""
from __future__ import annotations

import shutil
import subprocess

import pytest

from conftest import REPO


def test_abs_gt_for_any_limit(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    exe = tmp_path / "limits_host"
    subprocess.run([cxx, "-O2", "-std=gnu++17", "-ffp-contract=off", f"-I{REPO / 'spin-tracking_gb300' / 'csrc'}",
                    str(REPO / "tests" / "limits_host.cpp"), "-o", str(exe)], check=True, capture_output=True, text=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.strip() == "0"
