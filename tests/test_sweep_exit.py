"""How the CTAs of a cluster leave a windowed sweep after a wait has run out
(ccd_b200/csrc/sweep_exit.h), on a model of their barriers and messages (no GPU):
all of them reach the end of the cycle, and none leaves while bytes are on their
way to it."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_every_cta_leaves_after_what_was_sent_to_it_has_landed(tmp_path):
    exe = str(tmp_path / "exit_check")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=address,undefined", "-fno-sanitize-recover=all",
                        "-I" + os.path.join(ROOT, "ccd_b200", "csrc"),
                        os.path.join(ROOT, "tests", "native", "exit_check.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    r = subprocess.run([exe, "5000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.stdout[-2000:], r.stderr[-4000:])
    assert "all left in order" in r.stdout
