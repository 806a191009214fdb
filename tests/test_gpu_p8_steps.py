"""The shortened Mandelbulb<8> step (p8_de) against the step written operation
by operation: the packed grid kernel (de_grid_kernel 3) keeps the reference's
operations with CUDA's division and square roots, so the two grids agree bit
for bit or the shortened step is wrong.  The spans are those where it could
be: around the z axis and the origin (its axis bound, underflow), across the
planes y = 0 and z = 0, where its scaled coordinates lie about 2^-60, and
bailouts in and out of the range it is proven for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SPANS = {
    "cube": ((-1.2, -1.2, -1.2), (1.2, 1.2, 1.2)),
    "cube_off_centre": ((-1.1937, -1.2121, -1.1819), (1.2013, 1.1877, 1.2171)),
    "axis": ((-0.004, -0.004, 0.3), (0.004, 0.004, 0.9)),
    "axis_bound": ((0.00190, -0.0001, 0.5), (0.00200, 0.0001, 0.6)),
    "origin": ((-0.01, -0.01, -0.01), (0.01, 0.01, 0.01)),
    "origin_tiny": ((-1e-12, -1e-12, -1e-12), (1e-12, 1e-12, 1e-12)),
    "y_underflow": ((0.4, -1e-18, 0.3), (0.9, 1e-18, 0.8)),
    "z_underflow": ((0.4, 0.3, -1e-18), (0.9, 0.8, 1e-18)),
    "yz_denormal": ((0.4, -1e-38, -1e-38), (0.9, 1e-38, 1e-38)),
    "far": ((-9.0, -8.0, -7.0), (9.0, 10.0, 11.0)),
}


def grid(cg, variant, shape, span, res):
    import torch
    from cantucci_gb300 import _ffi
    lib = _ffi.load()
    _ffi.check(lib.cg_set_option(b"de_grid_kernel", variant))
    try:
        d = shape.span_grid(cg.Span(*span), res)
        torch.cuda.synchronize()
    finally:
        lib.cg_set_option(b"de_grid_kernel", 0)
    return d.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("iters,bailout", [(1, 2.5), (2, 2.5), (15, 2.5), (16, 5.0), (15, 16.0),
                                           (15, 17.0), (15, 0.001), (15, 1e30),
                                           (15, float("inf"))])
@pytest.mark.parametrize("name", sorted(SPANS))
def test_shortened_step_same_bits(cg, name, iters, bailout):
    s = cg.Mandelbulb(8, iters, bailout)
    ref = grid(cg, 3, s, SPANS[name], 32)
    for variant in (1, 2):
        assert np.array_equal(grid(cg, variant, s, SPANS[name], 32), ref), variant
    pts = [(0.0, 0.0, 0.0), (0.0, 0.0, 0.5), (np.inf, 0.1, 0.1), (0.1, np.nan, 0.2),
           (0.1, 0.2, -np.inf), (1e-30, 0.2, 0.3), (0.7, 0.0, -0.0)]
    d = s.batch_min_distance_from(np.array(pts, np.float32))
    assert d.shape == (7,)  # every special point ends


@pytest.mark.parametrize("bailout", [1e-6, 9e-7, 1e-15, 1e-21])
@pytest.mark.parametrize("name", ["cube", "origin", "origin_tiny", "yz_denormal"])
def test_tiny_bailouts_same_bits(cg, name, bailout):
    """Squares that escape a bailout about 2^-20 and below it: the last root is
    the shortened one only down to there."""
    s = cg.Mandelbulb(8, 15, bailout)
    ref = grid(cg, 3, s, SPANS[name], 32)
    for variant in (1, 2):
        assert np.array_equal(grid(cg, variant, s, SPANS[name], 32), ref), variant
