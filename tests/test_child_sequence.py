"""The order in which a traversal visits a node's hit children, on the CPU: near
to far with ties by slot, also where entry distances are infinite (a box at
infinity, a plane distance past the float range) and the ray has no end."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "rdna2-accel-raster_b200", "csrc")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="needs nvcc")
def test_child_sequence_matches_its_statement(tmp_path):
    exe = tmp_path / "child_sequence"
    r = subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-I", CSRC,
                        os.path.join(ROOT, "tests", "cpp", "child_sequence.cu"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
