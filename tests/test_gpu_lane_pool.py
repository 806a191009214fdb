"""Large point batches (k_de_points_pool, whose warps take new points as lanes
end) against the same points in batches small enough for the plain kernel: the
same bits for every estimator, for points without order, points side by side
and points on the surface, at sizes around a warp's groups and with ragged
ends."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMALL = 100_000


def shapes(cg):
    polar = cg.MandelbulbPolar(8.3, 15, 2.5, (0.2, 0.1, 0.0))
    return {"p8": cg.Mandelbulb(8, 15), "p8_it9": cg.Mandelbulb(8, 9),
            "int6": cg.Mandelbulb(6, 10), "polar": polar, "p8_fast": cg.Mandelbulb(8, 15).fast(),
            "int6_fast": cg.Mandelbulb(6, 12).fast(), "polar_fast": polar.fast(),
            "one_step": cg.Mandelbulb(8, 1), "sphere": cg.Sphere((0.1, 0.2, 0.3), 0.7)}


def points(order, n, shape):
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    p = torch.rand((n, 3), generator=g, device="cuda") * 2.6 - 1.3
    if order == "side_by_side":
        p = p[torch.argsort(p[:, 2])].contiguous()
        p[:, :2] *= 0.02
    if order == "surface":
        d = p / p.norm(dim=1, keepdim=True)
        p = d * 1.4
        for _ in range(12):
            for k in range(0, n, SMALL):
                p[k:k + SMALL] -= d[k:k + SMALL] * shape.batch_min_distance_from(
                    p[k:k + SMALL])[:, None].nan_to_num(0.0)
    if order == "special":
        p[::97] = 0.0
        p[5::101, 0] = float("nan")
        p[7::103, 1] = float("inf")
        p[11::107, :2] = 0.0
    return p


@pytest.mark.parametrize("order,n", [("random", 1_500_000), ("random", 1_500_031),
                                     ("side_by_side", 1_500_017), ("surface", 1_500_001),
                                     ("special", 1_500_007), ("random", 4_000_003),
                                     ("side_by_side", 2_500_017), ("surface", 2_500_001),
                                     ("special", 2_500_007)])
@pytest.mark.parametrize("name", ["p8", "p8_it9", "int6", "polar", "p8_fast", "int6_fast",
                                  "polar_fast", "one_step", "sphere"])
def test_large_batch_same_bits(cg, name, order, n):
    import torch
    shape = shapes(cg)[name]
    p = points(order, n, shape)
    big = shape.batch_min_distance_from(p)
    parts = [shape.batch_min_distance_from(p[k:k + SMALL]) for k in range(0, n, SMALL)]
    assert torch.equal(big.view(torch.int32), torch.cat(parts).view(torch.int32))
