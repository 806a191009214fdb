"""Large point batches of mixed order: parts in which neighbours lie side by
side beside parts in which they do not, so that the warps of the pool kernel
choose differently.  Every distance is written (the output is filled with
another pattern first) and has the bits that small batches give, which take the
one-point-per-thread kernel."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

SMALL = 100_000
UNWRITTEN = 0x12345678


def grid(n, row):
    """n points of a grid whose rows are `row` points long."""
    import torch
    i = torch.arange(n, device="cuda")
    side = int((n / row) ** 0.5) + 1
    z, y, x = i % row, i // row % side, i // row // side
    p = torch.stack([x / side, y / side, z / row], dim=1).float()
    return p * 2.4 - 1.2


def uniform(n):
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    return torch.rand((n, 3), generator=g, device="cuda") * 2.6 - 1.3


def vertices(cg, res):
    """The vertices of a mesh of the whole bulb, in id order."""
    import torch
    v = torch.empty((4_500_000, 7), device="cuda")
    ix = torch.empty(30_000_000, dtype=torch.int32, device="cuda")
    nv, _, _ = cg.Mesher().generate_device(cg.Span([-1.2] * 3, [1.2] * 3), cg.Mandelbulb(8, 15),
                                           res, v, ix, strict=False)
    return v[:nv, :3].contiguous()


def points(cg, order, n):
    import torch
    p = grid(n, 200)
    if order == "grid_then_uniform":
        p[100_000:] = uniform(n)[100_000:]
    elif order == "uniform_then_grid":
        p[:150_016] = uniform(n)[:150_016]
    elif order == "runs":  # 32 points of the grid, 32 without order, ...
        p = torch.where((torch.arange(n, device="cuda") // 32 % 2 == 0)[:, None], p, uniform(n))
    elif order == "nan":
        p[5 * 32 + 7, 1] = float("nan")
    elif order == "inf":
        p[11 * 32, 0] = float("inf")
    elif order == "far":
        p[901 * 32 + 31, 2] = 1e6
    elif order == "rows_of_20":
        p = grid(n, 20)
    elif order == "threshold":  # neighbours about as far apart as the kernel's limit
        p = uniform(n) * (0.25 / 2.6)
    elif order == "vertices":
        p = vertices(cg, 512)
        assert len(p) > 3_000_000
        p = p[:n].contiguous()
    return p


@pytest.mark.parametrize("n", [2_000_000, 3_700_011])
@pytest.mark.parametrize("order", ["grid_then_uniform", "uniform_then_grid", "runs", "nan", "inf",
                                   "far", "rows_of_20", "threshold", "vertices"])
def test_mixed_orders_write_every_distance(cg, order, n):
    import torch
    lib = cg.load()
    p = points(cg, order, n)
    n = p.shape[0]
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    wrong = {}
    for name, shape in (("p8", cg.Mandelbulb(8, 15)), ("p8_it9", cg.Mandelbulb(8, 9)),
                        ("int6", cg.Mandelbulb(6, 10)),
                        ("polar", cg.MandelbulbPolar(8.3, 15, 2.5, (0.2, 0.1, 0.0)))):
        out = torch.full((n,), UNWRITTEN, dtype=torch.int32, device="cuda")
        assert lib.cg_min_distance_from(C.byref(shape._cshape()), p.data_ptr(), n, out.data_ptr(),
                                        0, stream) == 0
        ref = torch.cat([shape.batch_min_distance_from(p[k:k + SMALL])
                         for k in range(0, n, SMALL)]).view(torch.int32)
        unwritten = int((out == UNWRITTEN).sum())
        if not torch.equal(out, ref):
            wrong[name] = (unwritten, int((out != ref).sum()))
    assert not wrong, "(unwritten, different) distances: %s" % wrong
