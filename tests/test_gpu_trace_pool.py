"""The pooled march (k_trace_pool: rays change lanes and warps while they march)
against one pixel per thread (trace_kernel 0): the same depths, bit for bit,
for every estimator, at images of one ray, of fewer rays than blocks, of ragged
sizes and of more rays than lanes, and at step limits around a round's."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def depth(cg, shape, w, h, steps, numerics, kernel):
    import torch
    from cantucci_gb300 import _ffi, fit
    lib = _ffi.load()
    cam = fit.camera(w, h)
    out = torch.full((h, w), 7.0, device="cuda")
    c = shape._cshape()
    _ffi.check(lib.cg_set_option(b"trace_kernel", kernel))
    try:
        _ffi.check(lib.cg_trace_depth(C.byref(c), C.byref(cam), steps, 1e-4, numerics,
                                      C.c_void_p(out.data_ptr()),
                                      C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        torch.cuda.synchronize()
    finally:
        lib.cg_set_option(b"trace_kernel", 1)
    return out


@pytest.mark.parametrize("w,h,steps", [(1, 1, 256), (3, 1, 64), (37, 29, 31), (128, 96, 256),
                                       (333, 250, 33), (800, 600, 100), (64, 64, 1), (50, 40, 0)])
@pytest.mark.parametrize("name", ["polar", "polar_fast", "p8", "p8_fast", "int6", "int6_fast",
                                  "sphere", "one_step"])
def test_pooled_march_same_depths(cg, name, w, h, steps):
    import torch
    shapes = {"polar": cg.MandelbulbPolar(8.3, 15, 2.5, (0.2, 0.1, 0.0)), "p8": cg.Mandelbulb(8, 15),
              "int6": cg.Mandelbulb(6, 10), "sphere": cg.Sphere((0.1, 0.0, 0.2), 0.9),
              "one_step": cg.Mandelbulb(8, 1)}
    shape = shapes[name.replace("_fast", "")]
    numerics = 1 if name.endswith("_fast") else 0
    a = depth(cg, shape, w, h, steps, numerics, 1)
    b = depth(cg, shape, w, h, steps, numerics, 0)
    assert torch.equal(a.view(torch.int32), b.view(torch.int32))
