"""The reverse-mode gradient over the long tape (every step's record, loops of 6
to 30 iterations) against the checkpointed tape (adjoint_ck 4: segments
recomputed).  Both sweep the same records through the same operations: the
outputs have the same bits.  And the batch product and its sums against the
per-point gradients."""
import numpy as np
import pytest

from cantucci_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def edge_points():
    p = W.uniform_points(5003, seed=5)
    p[:6] = [(0, 0, 0), (0, 0, 0.5), (0.7, 0, 0), (3.0, 0, 0), (1e-20, 0, 0.3), (1e-6, 1e-6, 0.6)]
    return p


@pytest.mark.parametrize("power,rot", [(8.0, (0, 0, 0)), (7.6, (0.2, -0.1, 0.3))])
@pytest.mark.parametrize("iters", [1, 2, 4, 5, 15, 19, 20, 21, 64])
def test_long_tape_matches_checkpoints(cg, iters, power, rot):
    import torch
    from cantucci_gb300 import _ffi
    from cantucci_gb300.autograd import de_grad
    lib = _ffi.load()
    p = torch.as_tensor(edge_points()).cuda()
    a = de_grad(p, power, rot, max_iters=iters)
    _ffi.check(lib.cg_set_option(b"adjoint_ck", 4))
    try:
        b = de_grad(p, power, rot, max_iters=iters)
    finally:
        lib.cg_set_option(b"adjoint_ck", 5)
    assert torch.equal(torch.isnan(a), torch.isnan(b))
    assert torch.equal(a.nan_to_num(1e9), b.nan_to_num(1e9))


@pytest.mark.parametrize("iters", [15, 20, 21])
@pytest.mark.parametrize("n", [1, 31, 5003])
def test_batch_product_matches_points(cg, n, iters):
    import torch
    from cantucci_gb300.autograd import de_grad, mandelbulb_de
    p = torch.as_tensor(edge_points()[-n:].copy()).cuda().requires_grad_(True)
    power = torch.tensor(8.0, requires_grad=True)
    rot = torch.zeros(3, requires_grad=True)
    w = torch.linspace(-1, 1, n, device="cuda")
    d = mandelbulb_de(p, power, rot, iters, 2.5)
    gp, gpow, grot = torch.autograd.grad((d * w).sum(), [p, power, rot])
    g = de_grad(p.detach(), 8.0, max_iters=iters)
    ref = w[:, None] * g
    assert torch.allclose(gp, ref[:, 1:4], rtol=1e-5, atol=0, equal_nan=True)
    terms = ref[:, 4:8].double()
    terms = torch.where(terms.isnan(), 0.0, terms)  # degenerate points are left out
    total, size = terms.sum(0), terms.abs().sum(0)
    got = torch.cat([gpow[None], grot]).double().cuda()
    assert ((got - total).abs() <= (n + 64) * 2.0 ** -24 * size + 1e-30).all()


@pytest.mark.parametrize("iters", [6, 9, 10, 17, 18, 30, 31])
@pytest.mark.parametrize("n", [1, 127, 129, 700001])
def test_tensor_memory_columns(cg, n, iters):
    """Where the columns per block change (9, 17 steps), at the edges of a block
    and with more groups than resident warps, on two streams at once."""
    import torch
    from cantucci_gb300 import _ffi
    from cantucci_gb300.autograd import de_grad
    lib = _ffi.load()
    p = torch.as_tensor(W.uniform_points(n, seed=11)).cuda()
    torch.cuda.synchronize()
    got = []
    for stream in (torch.cuda.Stream(), torch.cuda.Stream()):
        with torch.cuda.stream(stream):
            got.append(de_grad(p, 7.6, (0.2, -0.1, 0.3), max_iters=iters))
    torch.cuda.synchronize()
    _ffi.check(lib.cg_set_option(b"adjoint_ck", 4))
    try:
        ref = de_grad(p, 7.6, (0.2, -0.1, 0.3), max_iters=iters)
    finally:
        lib.cg_set_option(b"adjoint_ck", 5)
    for a in got:
        assert torch.equal(torch.isnan(a), torch.isnan(ref))
        assert torch.equal(a.nan_to_num(1e9), ref.nan_to_num(1e9))
