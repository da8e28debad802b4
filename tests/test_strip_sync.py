"""Memory order between the warps of the 2D strips schedule (pfast_gb300/csrc/strip_sync.h), on the
CPU: tests/native/strip_sync_check.cpp runs its publish and wait over vector clocks."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_strips_order_every_lane(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "strip_sync_check")
    subprocess.run([gxx, "-std=c++17", "-O2", "-I", os.path.join(ROOT, "pfast_gb300", "csrc"),
                    os.path.join(HERE, "native", "strip_sync_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.count("ok ") == 4, out.stdout
