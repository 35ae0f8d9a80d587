"""The tests of the small meshes' shared launches and of the edge tiles once more against the
checked library (test_gpu_checked.py says what that is), in a child process: no index is out of
range there, and the checks change no bits."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_small_meshes_and_tiles_under_the_checked_build():
    sys.path.insert(0, os.path.join(ROOT, "dg-rain_b200"))
    import build

    assert os.path.exists(build.build_checked())
    res = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-m", "gpu", "tests/test_gpu_small_meshes.py",
                          "tests/test_gpu_edge_tiles.py"],
                         cwd=ROOT, env=dict(os.environ, DGRAIN_LIBRARY="checked"), capture_output=True, text=True)
    tail = (res.stdout + res.stderr)[-3000:]
    assert res.returncode == 0 and " passed" in res.stdout, tail
