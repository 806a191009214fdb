"""Step 1 in core units and faces (grid_units.cuh), with the work queue (through
the mesher) and in strides (cg_de_span_grid), against one corner per thread in
row order (de_grid_kernel 1): the same distances, bit for bit, and the same
sign words (through the indices), at every resolution that takes them -- 32 and
64 (one unit per warp), 256 and up (persistent warps) -- and at 16 and 128, which
do not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("power,iters,res", [(8, 15, 16), (8, 15, 32), (8, 7, 64), (6, 10, 64),
                                             (8, 15, 128), (8, 15, 256), (8, 4, 512), (6, 4, 256)])
def test_units_match_row_order(cg, power, iters, res):
    import torch
    from cantucci_gb300 import _ffi
    lib = _ffi.load()
    shape = cg.Mandelbulb(power, iters, 2.5)
    span = cg.Span([-1.21, -1.2, -1.19], [1.2, 1.22, 1.2])
    room = 24 * res * res + 4096
    got = {}
    m = cg.Mesher(0)
    try:
        for kernel in (0, 1):
            _ffi.check(lib.cg_set_option(b"de_grid_kernel", kernel))
            d = shape.span_grid(span, res)
            v = torch.zeros((room, 7), device="cuda")
            i = torch.zeros(8 * room, dtype=torch.int32, device="cuda")
            nv, ni, _ = m.generate_device(span, shape, res, v, i, strict=False)
            dists = m.last_dists()
            assert torch.equal(dists.view(torch.int32), d.view(torch.int32))
            got[kernel] = (d, nv, ni, v, i)
    finally:
        lib.cg_set_option(b"de_grid_kernel", 0)
        m.close()
    a, b = got[0], got[1]
    assert a[1:3] == b[1:3]
    for x, y in ((a[0], b[0]), (a[3], b[3]), (a[4], b[4])):
        assert torch.equal(x.view(torch.int32), y.view(torch.int32))
