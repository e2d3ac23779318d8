"""The windowed sweep's plan (ccd_b200/csrc/window_plan.cpp) against a pairwise
comparison of the columns, under AddressSanitizer and UBSan (no GPU): which
columns share a row, and which entries each CTA owns."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_window_plan_matches_pairwise_comparison(tmp_path):
    exe = str(tmp_path / "window_check")
    csrc = os.path.join(ROOT, "ccd_b200", "csrc")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=address,undefined", "-fno-sanitize-recover=all",
                        "-I" + csrc, os.path.join(ROOT, "tests", "native", "window_check.cpp"),
                        os.path.join(csrc, "window_plan.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    r = subprocess.run([exe, "300"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.stdout[-2000:], r.stderr[-4000:])
    assert "identical" in r.stdout


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_quotient_step_matches_the_closed_forms(tmp_path):
    """The windowed sweep's step against newton_prior_delta_l, infinities and
    not-a-numbers included."""
    exe = str(tmp_path / "step_check")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I" + os.path.join(ROOT, "ccd_b200", "csrc"),
                        os.path.join(ROOT, "tests", "native", "step_check.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout[-2000:]
    assert "identical" in r.stdout
