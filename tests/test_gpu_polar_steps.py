"""The shortened exact step of the polar maps (polar_radius, powi_pair, no
angles in the last step) against the loop state of the step written operation
by operation (cg_mandelbulb_state): the distance formed from that state's r and
dr, at powers around the bits of powi, at bailouts in and out of the range of
the shortened operations, and at points where they do not apply (z axis,
origin, tiny and non-finite coordinates)."""
import ctypes as C

import numpy as np
import pytest

from cantucci_gb300 import workloads as W

pytestmark = pytest.mark.gpu

EDGE = [(0, 0, 0), (0, 0, 0.5), (0, 0, -0.7), (1e-38, 0, 0.4), (1e-20, 1e-20, 1e-20),
        (0.3, -0.0, 1e-40), (1e-31, 1e-31, 0.6), (5e-10, 3e-10, 1e-9), (2e5, 0.1, 0.1),
        (np.inf, 0.1, 0.1), (0.1, np.nan, 0.2), (0.7, 0.1, -np.inf)]
# |ln r| within 1 ulp of CUDA's logf against the correctly rounded value, and
# two roundings on each side of the product and the quotient: under 6 half ulps
ULPS = 4


def state(shape, pts):
    import torch
    from cantucci_gb300 import _ffi
    out = torch.empty((len(pts), 4), dtype=torch.float32, device="cuda")
    p = torch.as_tensor(pts).cuda()
    s = shape._cshape()
    _ffi.check(_ffi.load().cg_mandelbulb_state(C.byref(s), C.c_void_p(p.data_ptr()), len(pts),
                                               C.c_void_p(out.data_ptr()), None))
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("iters,bailout", [(1, 2.5), (2, 2.5), (15, 2.5), (10, 0.001), (10, 3e6),
                                           (10, float("inf"))])
@pytest.mark.parametrize("P", [1, 2, 3, 6, 7, 9, 10, 16])
def test_integer_power_distance_follows_state(cg, P, iters, bailout):
    shape = cg.Mandelbulb(P, iters, bailout)
    pts = np.concatenate([np.array(EDGE, np.float32), W.uniform_points(20011, seed=40 + P),
                          W.uniform_points(1013, seed=60 + P) * np.float32(1e-3)])
    d = shape.batch_min_distance_from(pts)
    st = state(shape, pts)
    with np.errstate(all="ignore"):
        r, dr = st[:, 0].astype(np.float64), st[:, 1].astype(np.float64)
        ref = 0.5 * np.log(r) * r / dr
    ok = np.isfinite(ref) & (np.abs(ref) > 1e-30) & (np.abs(ref) < 1e30) & (r < 1e18) & (dr < 1e30)
    assert ok.any()
    err = np.abs(d[ok].astype(np.float64) - ref[ok]) / np.abs(ref[ok])
    assert err.max() <= ULPS * 2.0 ** -23
    assert np.array_equal(np.isnan(d), np.isnan(ref))
