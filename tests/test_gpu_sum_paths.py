"""The batch product, the surface term and the depth map's backward pass on both
sides of every line of their dispatch: loops of up to 5 steps and of 31 and more
take the checkpointed tape, those between the long one, and the surface term has
a third form with adjoint_recompute 1.  Each against the per-point gradients of
the same tape (cg_de_grad), added up in double; a sum differs from that only by
the float it is returned in and, for the product, by the float of each term."""
import ctypes as C

import pytest

from cantucci_gb300 import workloads as W

pytestmark = pytest.mark.gpu

ITERS = [1, 5, 6, 30, 31, 64]
ULP = 2.0 ** -24


def points(n):
    import torch
    p = W.uniform_points(max(n, 8), seed=17)
    p[:4] = [(0, 0, 0), (0, 0, 0.5), (0.7, 0, 0), (1e-20, 0, 0.3)]
    return torch.as_tensor(p[:n].copy()).cuda()


@pytest.mark.parametrize("iters", ITERS)
@pytest.mark.parametrize("n", [33, 129, 20011])
def test_batch_product(cg, n, iters):
    import torch
    from cantucci_gb300.autograd import de_grad, mandelbulb_de
    p = points(n).requires_grad_(True)
    power, rot = torch.tensor(7.7, requires_grad=True), torch.tensor([0.1, -0.2, 0.3],
                                                                    requires_grad=True)
    w = torch.linspace(-1, 1, n, device="cuda")
    gp, gpow, grot = torch.autograd.grad(mandelbulb_de(p, power, rot, iters, 2.5), [p, power, rot],
                                         w)
    ref = w[:, None] * de_grad(p.detach(), 7.7, rot.tolist(), iters)
    assert torch.equal(gp.nan_to_num(1e9), ref[:, 1:4].nan_to_num(1e9))
    t = ref[:, 4:8].double()
    t = torch.where(t.isnan(), 0.0, t)  # degenerate points are left out
    got = torch.cat([gpow[None], grot]).double().cuda()
    assert ((got - t.sum(0)).abs() <= 4 * ULP * t.abs().sum(0) + 1e-37).all()


@pytest.mark.parametrize("iters", ITERS)
@pytest.mark.parametrize("recompute", [0, 1])
@pytest.mark.parametrize("n", [33, 20011])
def test_surface_term(cg, n, recompute, iters):
    import torch
    from cantucci_gb300 import fit
    from cantucci_gb300.autograd import de_grad
    lib, p = cg.load(), points(n)
    power, rot = torch.tensor(7.7, requires_grad=True), torch.tensor([0.1, -0.2, 0.3],
                                                                    requires_grad=True)
    assert lib.cg_set_option(b"adjoint_recompute", recompute) == 0
    try:
        loss = fit.surface_loss(power, rot, p, max_iters=iters, cap=1.0)
        g = de_grad(p, 7.7, rot.tolist(), iters).double()
    finally:
        lib.cg_set_option(b"adjoint_recompute", 0)
    gpow, grot = torch.autograd.grad(loss, [power, rot])
    ok = torch.isfinite(g).all(dim=1)
    keep = ok & (g[:, 4:8].abs().amax(dim=1) <= 1.0)
    m = max(int(ok.sum()), 1)
    t = torch.cat([g[ok, 0].abs().sum()[None],
                   (torch.sign(g[keep, :1]) * g[keep, 4:8]).sum(0)]) / m
    size = torch.cat([t[:1], g[keep, 4:8].abs().sum(0) / m])
    got = torch.cat([loss.detach()[None], gpow[None].cuda(), grot.cuda()]).double()
    assert ((got - t).abs() <= 4 * ULP * size + 1e-37).all()


def backward(cg, cam, depth, g, iters):
    import torch
    from cantucci_gb300.autograd import _shape
    out = torch.empty(4, device="cuda")
    shape = _shape(7.7, [0.1, -0.2, 0.3], iters, 2.5)
    assert cg.load().cg_trace_backward(C.byref(shape), C.byref(cam), depth.data_ptr(),
                                       g.data_ptr(), out.data_ptr(),
                                       torch.cuda.current_stream().cuda_stream) == 0
    return out


@pytest.mark.parametrize("iters", ITERS)
def test_depth_backward_of_one_pixel(cg, iters):
    """A camera whose only ray is -z: the point at depth t is known exactly."""
    import torch
    from cantucci_gb300 import fit
    from cantucci_gb300.autograd import de_grad
    cam = fit.camera(1, 1)
    cam.eye[0], cam.eye[1] = cam.target[0], cam.target[1] = 0.25, 0.375
    g = torch.full((1, 1), 0.5, device="cuda")
    for t in (1.0, 1.4, 1.6, 1.9):
        depth = torch.full((1, 1), t, device="cuda")
        p = torch.tensor([[0.25, 0.375, 2.5 - float(depth)]], device="cuda")
        o = de_grad(p, 7.7, [0.1, -0.2, 0.3], iters)[0].double()
        ref = 0.5 * -o[4:8] / -o[3]
        got = backward(cg, cam, depth, g, iters).double()
        assert ((got - ref).abs() <= 4 * ULP * ref.abs()).all()


@pytest.mark.parametrize("iters", ITERS[1:])  # (one step has no surface)
def test_depth_backward_adds_its_pixels(cg, iters):
    import torch
    from cantucci_gb300 import fit
    cam = fit.camera(96, 72)
    depth = fit.render(7.7, (0.1, -0.2, 0.3), cam, max_iters=iters)
    hit = (depth > 0).nonzero()
    assert len(hit) > 100
    hit = hit[:: len(hit) // 40]
    g, one = torch.zeros_like(depth), []
    for k, (y, x) in enumerate(hit.tolist()):
        single = torch.zeros_like(depth)
        g[y, x] = single[y, x] = 0.3 + 0.1 * k
        one.append(backward(cg, cam, depth, single, iters).double())
    one = torch.stack(one)
    got = backward(cg, cam, depth, g, iters).double()
    size = one.abs().sum(0) + got.abs()
    assert torch.isfinite(got).all() and (got != 0).any()
    assert ((got - one.sum(0)).abs() <= 1.01 * ULP * size + 1e-37).all()
