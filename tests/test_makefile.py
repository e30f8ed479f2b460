"""The library's Makefile rebuilds every object whose sources include a header
that changed: an object left as it was would keep the old inline code."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "rdna2-accel-raster_b200", "csrc")


def included(path, seen):
    """The repository's headers that a source reaches."""
    for name in re.findall(r'^\s*#include "([^"]+)"', open(path).read(), re.M):
        p = os.path.normpath(os.path.join(os.path.dirname(path), name))
        if p not in seen:
            seen.add(p)
            included(p, seen)
    return seen


@pytest.mark.skipif(shutil.which("make") is None, reason="needs make")
def test_objects_depend_on_the_headers_they_include(tmp_path):
    sources = [f for f in os.listdir(CSRC) if f.endswith((".cu", ".cpp"))]
    # a tree in which everything is built
    for f in sources:
        (tmp_path / f.rsplit(".", 1)[0]).with_suffix(".o").touch()
    headers = {}
    for f in sources:
        for h in included(os.path.join(CSRC, f), set()):
            headers.setdefault(h, set()).add(f)
    assert any(h.endswith("collapse_core.cuh") for h in headers)
    for h, users in headers.items():
        out = subprocess.run(["make", "-n", "-C", CSRC, f"BUILD={tmp_path}", f"OUT={tmp_path}/librq.so", "-W",
                              os.path.relpath(h, CSRC)], capture_output=True, text=True, check=True).stdout
        stale = [f for f in users if f"-c {f} " not in out]
        assert not stale, f"{os.path.basename(h)}: {stale} would stay as they are"
