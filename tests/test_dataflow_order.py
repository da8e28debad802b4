"""Memory order of the 3D dataflow kernel's queue (pfast_gb300/csrc/dataflow_queue.h), on the CPU:
tests/native/dataflow_order_check.cpp runs the queue's own functions over a memory with vector clocks
and checks that a lane which starts on a tile has seen what the tiles it waited for wrote, for the
queue of a block and of a cluster.  (On the GPU a missing order shows only by chance, as a wrong
value.)"""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_queue_orders_writes_before_reads(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "dataflow_order_check")
    subprocess.run([gxx, "-std=c++17", "-O2", "-I", os.path.join(ROOT, "pfast_gb300", "csrc"),
                    os.path.join(HERE, "native", "dataflow_order_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and "FAIL" not in out.stdout and out.stdout.count("ok ") == 6, out.stdout
