"""The tables that batches and instance scenes upload are on the device before
a kernel on any stream reads them.  capi_batch.cpp and tlas.cpp run on the CPU
against a model of CUDA's stream ordering (tests/cpp/upload_order.cpp)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "rdna2-accel-raster_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")
CXX = shutil.which("g++")


@pytest.mark.skipif(CXX is None, reason="needs g++")
def test_tables_are_written_before_they_are_read(tmp_path):
    exe = tmp_path / "upload_order"
    cmd = [CXX, "-std=c++17", "-O1", "-I", CSRC, "-I", os.path.join(CUDA, "include"),
           os.path.join(ROOT, "tests", "cpp", "upload_order.cpp"), os.path.join(CSRC, "capi_batch.cpp"),
           os.path.join(CSRC, "tlas.cpp"), "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
