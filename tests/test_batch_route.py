"""The batch engine's dispatch (ccd_b200/csrc/batch_route.h), without a GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_batch_routes(tmp_path):
    exe = str(tmp_path / "batch_route_check")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I" + os.path.join(ROOT, "ccd_b200", "csrc"),
                        os.path.join(ROOT, "tests", "native", "batch_route_check.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout[-2000:]
    assert "all routes as expected" in r.stdout
