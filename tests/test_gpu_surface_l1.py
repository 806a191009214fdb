"""cg_surface_l1 (one fused pass) against the same sums formed from the
per-point gradients (cg_de_grad) in double: counts, the cap's selection and
degenerate points alike; the sums differ only by the float they are returned
in, 4 * 2^-24 of the largest term sum."""
import numpy as np
import pytest

from cantucci_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("iters", [1, 15, 20, 21])
@pytest.mark.parametrize("cap", [0.0, 1.0])
@pytest.mark.parametrize("n", [0, 1, 63, 65, 20011])
def test_fused_surface_loss(cg, n, cap, iters):
    import torch
    from cantucci_gb300 import fit
    from cantucci_gb300.autograd import de_grad
    p = W.uniform_points(max(n, 1), seed=3)[:n]
    if n > 64:
        p[:3] = [(0, 0, 0), (0, 0, 0.5), (0.7, 0, 0)]  # derivatives that are not finite
    pts = torch.as_tensor(p).cuda().reshape(-1, 3)
    power = torch.tensor(8.2, requires_grad=True)
    rot = torch.tensor([0.1, -0.2, 0.3], requires_grad=True)
    loss = fit.surface_loss(power, rot, pts, max_iters=iters, cap=cap)
    gpow, grot = torch.autograd.grad(2.0 * loss, [power, rot])
    g = de_grad(pts, float(power), rot.tolist(), iters).double()
    ok = torch.isfinite(g).all(dim=1)
    m = max(int(ok.sum()), 1)
    keep = ok & (g[:, 4:8].abs().amax(dim=1) <= cap) if cap > 0 else ok
    terms = torch.sign(g[keep, :1]) * g[keep, 4:8]
    ref = torch.cat([g[ok, 0].abs().sum()[None], 2.0 * terms.sum(0)]).cpu() / m
    got = torch.cat([loss.detach().cpu()[None], gpow[None], grot]).double()
    size = torch.cat([ref[:1].abs(), 2.0 * terms.abs().sum(0).cpu() / m])
    assert ((got - ref).abs() <= 4 * 2.0 ** -24 * size + 1e-37).all()
    assert loss.is_cuda and loss.ndim == 0 and gpow.device == power.device
