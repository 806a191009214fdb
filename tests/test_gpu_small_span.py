"""The small-span kernels (k_de_grid_small, k_rows_cluster, k_place_spread,
k_quad_emit_fine) against the batched mesher's row-by-row kernels and one
vertex per thread: the same vertices and indices, bit for bit, from the
smallest grid to the largest they take, without a surface, with few vertices
(four to a warp) and with many (nine), and cut at small capacities."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SPANS = {"cube": ((-1.2, -1.2, -1.2), (1.2, 1.2, 1.2)),
         "surface": ((0.55, -0.35, 0.45), (0.95, 0.05, 0.85)),
         "dense": ((0.60, 0.58, -0.02), (0.66, 0.64, 0.04)),
         "outside": ((1.5, 1.5, 1.5), (1.7, 1.7, 1.7)),
         "inside": ((0.1, 0.1, 0.1), (0.2, 0.2, 0.2))}


@pytest.mark.parametrize("res", [2, 4, 8, 16, 32, 64])
@pytest.mark.parametrize("name", sorted(SPANS))
@pytest.mark.parametrize("power,iters", [(8, 15), (8, 12), (6, 10)])
def test_small_span_matches_batch(cg, name, res, power, iters):
    import torch
    from cantucci_gb300.batch import BatchMesher
    lo, hi = SPANS[name]
    shape = cg.Mandelbulb(power, iters, 2.5)
    b = BatchMesher(np.array([lo + hi], np.float32), [res])
    v, i = b.run(shape).mesh(0)
    m = cg.Mesher(0)
    try:
        for cap in (res ** 3, max(len(v) // 2, 1)):
            dv = torch.full((cap + 1, 7), 7.0, device="cuda")
            di = torch.full((18 * res ** 3 + 1,), 7, dtype=torch.int32, device="cuda")
            args = (cg.Span(lo, hi), shape, res, dv[:cap], di)
            try:  # (a lerp failure, reported first, is not raised)
                nv, ni, _ = m.generate_device(*args, strict=False)
                assert (nv, ni) == (len(v), len(i))
            except cg.CantucciError:
                assert cap < len(v)
            k = min(cap, len(v))
            assert np.array_equal(dv[:k].cpu().numpy().view(np.uint32), v[:k].view(np.uint32))
            assert (dv[cap] == 7.0).all()
            assert np.array_equal(di[:len(i)].cpu().numpy().view(np.uint32), i)
            assert int(di[-1]) == 7
    finally:
        m.close()
        b.close()
