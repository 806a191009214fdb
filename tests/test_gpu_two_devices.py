"""Spans up to res 64 mesh on every GPU of a process: their 16-CTA cluster launch
needs an attribute that a kernel has per device, so it is set on each one that
meshes.  Two devices are made of one GPU by a preloaded shim (cpp/two_devices.cpp)
that prints where the attribute is set."""
import os
import shutil
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = """
import cantucci_gb300 as cg

lib = cg.load()
span, shape = cg.Span([-1.2] * 3, [1.2] * 3), cg.Mandelbulb(8, 15)
assert lib.cg_set_option(b"mesh_graphs", %d) == 0
out = []
for device in (0, 1, 0):
    m = cg.Mesher(device)
    for res in (16, 64):
        v, ix, nv, ni, _ = m.generate(span, shape, res, strict=False)
        out.append((device, res, v[:nv].tobytes(), ix[:ni].tobytes()))
    m.close()
assert [o[1:] for o in out[:2]] == [o[1:] for o in out[2:4]] == [o[1:] for o in out[4:]]
"""


@pytest.mark.parametrize("graphs", [1, 0])
def test_cluster_attribute_on_each_device(cg, tmp_path, graphs):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    nvcc = os.path.realpath(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc")
    shim = str(tmp_path / "two_devices.so")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I",
                        os.path.join(os.path.dirname(os.path.dirname(nvcc)), "include"),
                        os.path.join(ROOT, "tests", "cpp", "two_devices.cpp"), "-o", shim, "-ldl"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([sys.executable, "-c", CHILD % graphs], cwd=ROOT, capture_output=True,
                       text=True, timeout=300, env={**os.environ, "LD_PRELOAD": shim})
    assert r.returncode == 0, r.stderr
    assert set(r.stdout.splitlines()) == {"device 0 cluster 1", "device 1 cluster 1"}
