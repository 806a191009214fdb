"""The shares that the warps of the point pool walk hold every point of a batch
exactly once, whatever sizes each warp takes its points in (host code, no GPU)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    out = str(tmp_path_factory.mktemp("pool") / "pool_walk")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-I",
                        os.path.join(ROOT, "cantucci_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "pool_walk.cpp"), "-o", out],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


@pytest.mark.parametrize("blocks", [1, 2, 3, 7, 304, 2432, 3040])
@pytest.mark.parametrize("n", [1, 31, 33, 128, 4095, 50017, 389120, 2_000_000, 3_700_011])
def test_every_point_once(walk, blocks, n):
    r = subprocess.run([walk, str(blocks), str(n), str(blocks + n)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
