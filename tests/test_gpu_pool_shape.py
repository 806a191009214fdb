"""The launch shape of a large point batch is that of its estimator and its size,
whichever estimator the process used first: read from the kernel node of a
captured graph, in processes that call the estimators in opposite orders."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes as C, sys
import torch
import cantucci_gb300 as cg


class KernelParams(C.Structure):
    _fields_ = [("func", C.c_void_p), ("grid", C.c_uint * 3), ("block", C.c_uint * 3),
                ("shared", C.c_uint), ("params", C.c_void_p), ("extra", C.c_void_p)]


lib, rt = cg.load(), C.CDLL("libcudart.so.13")
shapes = {"p8": cg.Mandelbulb(8, 15), "p8_it9": cg.Mandelbulb(8, 9), "int6": cg.Mandelbulb(6, 10),
          "polar": cg.MandelbulbPolar(8.3, 15)}
p = torch.zeros((9_000_000, 3), device="cuda")
out = torch.empty(9_000_000, device="cuda")
stream = torch.cuda.Stream()
st = C.c_void_p(stream.cuda_stream)
for name in sys.argv[1:]:
    for n in (1_000_000, 1_300_000, 1_700_000, 3_000_000, 9_000_000):
        graph, count, node, k = C.c_void_p(), C.c_size_t(1), C.c_void_p(), KernelParams()
        assert rt.cudaStreamBeginCapture(st, 2) == 0
        assert lib.cg_min_distance_from(C.byref(shapes[name]._cshape()), p.data_ptr(), n,
                                        out.data_ptr(), 0, st) == 0
        assert rt.cudaStreamEndCapture(st, C.byref(graph)) == 0
        assert rt.cudaGraphGetNodes(graph, C.byref(node), C.byref(count)) == 0 and count.value == 1
        assert rt.cudaGraphKernelNodeGetParams(node, C.byref(k)) == 0
        assert rt.cudaGraphDestroy(graph) == 0
        print(name, n, k.grid[0], k.block[0])
"""


def shapes(order):
    r = subprocess.run([sys.executable, "-c", CHILD, *order], cwd=ROOT, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    return sorted(r.stdout.splitlines())


def test_launch_shape_does_not_depend_on_earlier_calls(cg):
    order = ["p8", "int6", "polar", "p8_it9"]
    a, b = shapes(order), shapes(order[::-1])
    assert len(a) == 20 and a == b
