"""The pole step's roundings and product scans on the host, from the kernels' own source (tests/pole_host_check.cu, compiled by
nvcc, host code only): pm_limbs and pm_round of the tensor-core form for every limb count (the two usual lengths of a sum, the
general one, carries to the top, values planted next to midpoints), mac_signed_win and mac_signed_high of the CUDA-core
kernels."""
import os
import subprocess

import pytest

from blocksvibe_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def report(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("pole") / "pole_host_check")
    subprocess.run([build._nvcc(), *build.ARCH, "-O1", "-std=c++17", "-I", build.CSRC, "-o", exe,
                    os.path.join(HERE, "pole_host_check.cu")], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=600).stdout
    return {(name, int(L)): (int(n), int(bad)) for name, L, n, bad in (line.split() for line in out.strip().splitlines())}


@pytest.mark.parametrize("L", build.LIMBS)
@pytest.mark.parametrize("check", ["limbs", "round", "win", "high"])
def test_no_failures(report, check, L):
    cases, failures = report[check, L]
    assert cases > 0 and failures == 0


@pytest.mark.parametrize("L", build.LIMBS)
def test_redo_where_a_midpoint_is_near(report, L):
    redone, without_reason = report["redo", L]
    assert without_reason == 0 and redone < 20000
    assert redone > 100 or L < 14                            # nothing is dropped for the shortest numbers
